"""The softmax warps meet at a named barrier, which has no limit. A warp whose bounded wait has given up leaves only behind a meeting at
which all four learn of it: with any wait of any warp giving up, alone or with others, none is left at the barrier."""

import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
WALKS = [  # chunks of a block's tokens
    [1], [0], [10], [2, 2], [0, 0, 1], [1, 0, 1], [1, 1, 1, 0, 0, 3], [3, 0, 0, 2, 1], [2, 10, 1, 0], [0, 4, 0],
]


def role(source):
    start = source.index("template <int kFormat>\n__device__ void softmax_role(")
    text = source[start:source.index("// ---- kernel and launch", start)]
    # what a thread of a warp hands to the barrier, as a function of its lane
    text, found = re.subn(r"named_barrier_count\((.*), (failed [^;]*)\); };", r"named_barrier_count(\1, [&](int lane) -> bool { return \2; }); };", text)
    assert found == 1
    return source[source.index("enum Bar {"):source.index("};", source.index("enum Bar {")) + 2] + "\n" + text


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    def build(source):
        folder = tmp_path_factory.mktemp("role")
        (folder / "role.inc").write_text(role(source))
        subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-pthread", f"-I{folder}", str(ROOT / "tests/softmax_exits.cpp"),
                        "-o", str(folder / "exits")], check=True)
        return folder / "exits"
    return build


def runs():
    for chunks in WALKS:
        waits = sum(chunks) * 2 + 2 * len(chunks) + 1  # more than a warp can have
        for rescale in (0, 0xFFFFFFFF, 0x5A5A5A5A):
            for mode in (0, 1, 2):
                for warp in range(4):
                    for wait in range(waits):
                        yield f"{mode} {len(chunks)} {' '.join(map(str, chunks))} {rescale} {warp} {wait}\n"


def test_no_warp_is_left_at_a_barrier_when_waits_give_up(program):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    source = (ROOT / "ascendflow_b200/csrc/sparse_mla_tcgen05.cuh").read_text()
    lines = "".join(runs())
    result = subprocess.run([program(source)], input=lines, capture_output=True, text=True, timeout=300)
    assert result.stdout == "ok\n", result.stdout


@pytest.mark.parametrize("line", ["failed = true; meet(true); return;", "if (met >= kGivenUp) return;", "  meet(false);  // with a warp that"])
def test_a_way_out_that_misses_a_barrier_is_found(program, line):
    """The same on a text of the role in which one of its exits forgets the others."""
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    source = (ROOT / "ascendflow_b200/csrc/sparse_mla_tcgen05.cuh").read_text()
    assert source.count(line) == 1
    broken = source.replace(line, {"f": "failed = true; return;", "i": ""}.get(line[0], "//"))
    result = subprocess.run([program(broken)], input="".join(runs()), capture_output=True, text=True, timeout=300)
    assert result.stdout.startswith("left behind"), result.stdout
