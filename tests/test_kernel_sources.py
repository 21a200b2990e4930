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


def test_waits_for_other_blocks_acquire_at_cluster_scope():
    """What other blocks complete (by remote stores and copies) is waited for at their scope; the sender of P waits for its
    own block's warps only."""
    source = (CSRC / "sparse_mla_team.cuh").read_text()
    remote = set(re.findall(r"cluster_address\(sm\.bar\((\w+)", source))
    assert remote == {"kMaxima", "kP0"}
    for barrier in remote:
        waits = re.findall(rf"(\w+_wait(?:<true>)?)\(sm\.bar\({barrier}([^)]*)\)", source)
        assert waits
        for wait, item in waits:
            assert wait.endswith("<true>") or item == " + item", (barrier, wait, item)
    wrappers = (CSRC / "tcgen05_ptx.cuh").read_text()
    body = wrappers[wrappers.index("bool mbar_try_wait("):]
    assert "mbarrier.try_wait.parity.acquire.cluster." in body[: body.index("\n}\n")]


def test_slots_are_resolved_by_one_routine():
    """The rule from slot to row stands once beside the tcgen05 kernels, and all forms of resolving a token run it."""
    source = (CSRC / "sparse_mla_tcgen05.cuh").read_text()
    assert source.count("report(p, kStatusBadPage") == 1
    assert "kStatusBadPage" not in (CSRC / "sparse_mla_team.cuh").read_text()
