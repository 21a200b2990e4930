"""Rules of the kernels' sources that no run on a GPU can show to hold."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "ascendflow_b200" / "csrc"


@pytest.mark.parametrize("name,barriers", [("sparse_mla_tcgen05.cuh", ("kKvFull0",)), ("sparse_mla_team.cuh", ("kTile0", "kSlices0"))])
def test_operands_copied_by_cp_async_are_fenced_before_the_tensor_core_reads_them(name, barriers):
    """Whoever waits on a barrier that `cp_async_arrive` completes does so through `wait_for_copies`, which has the fence."""
    source = (CSRC / name).read_text()
    copied = set(re.findall(r"cp_async_arrive\(sm\.bar\((\w+)", source))
    assert copied == set(barriers)
    for barrier in copied:
        waits = re.findall(rf"(\w+)\(sm\.bar\({barrier}[^;{{]*abort_flag\)", source)
        assert waits and set(waits) == {"wait_for_copies"}
    common = (CSRC / "sparse_mla_tcgen05.cuh").read_text()
    body = common[common.index("bool wait_for_copies("):]
    assert "fence_proxy_async();" in body[: body.index("\n}\n")]
