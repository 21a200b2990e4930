"""The index selection's block on the CPU (`select_block.cpp`): results and stores out of range for rows that are listed whole and whose
threshold lies among the lowest keys (masks, NaNs with a sign). A fault there is shown here and not on a GPU."""

import re
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
MASKS = (0xFF800000, 0xFF7FFFFF, 0xFFFFFFFF, 0xFF800001)  # -inf, the lowest finite value, NaNs with a sign
HIGHEST = (1.5, 3.0, 6.0, 12.0, -1.0)                     # neighbouring binades: where the bins of the distance end


def kernel_text(source):
    text = source[source.index("// Monotone map"):source.index("// One warp per new row")]
    for name in ("prefetch_l2", "shared_add_if", "shared_or_if", "copy_word"):  # one instruction each: the CPU has its own
        text, found = re.subn(rf"__device__ __forceinline__ void {name}\([^)]*\) {{\n  asm volatile\(.*\);\n}}\n", "", text)
        assert found == 1, name
    text, found = re.subn(r'asm volatile\("cp\.async\.wait_all;\\n" ::: "memory"\);', "wait_for_words();", text)
    assert found == 2 and "asm" not in text
    rule = source[source.index("int launch_sparse_mla_topk_indices("):]
    return text + rule[:rule.index("\n}\n") + 3]


@pytest.fixture(scope="module")
def select(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    folder = tmp_path_factory.mktemp("block")
    (folder / "select.inc").write_text(kernel_text((ROOT / "ascendflow_b200/csrc/sparse_mla_neighbours.cu").read_text()))
    subprocess.run(["g++", "-std=c++17", "-O2", "-w", f"-I{folder}", str(ROOT / "tests/select_block.cpp"), "-o", str(folder / "block")], check=True)

    def run(rows, lengths, bits):
        """A call of `rows` rows of which the first len(bits) are looked at."""
        head = np.array([rows, bits.shape[1], len(bits)], dtype=np.int32).tobytes()
        result = subprocess.run([folder / "block"], input=head + np.asarray(lengths, dtype=np.int32).tobytes() + bits.tobytes(), capture_output=True, timeout=300)
        assert result.returncode == 0, result.stderr.decode()
        return np.frombuffer(result.stdout, dtype=np.int32).reshape(len(bits), 512)
    return run


def best(bits):
    """The 512 highest by their keys, the lower index first among equal ones, in index order."""
    key = np.where(bits >> 31, ~bits, bits | 0x80000000)
    out = np.full(512, -1, dtype=np.int32)
    picked = np.sort(np.argsort(~key, kind="stable")[:512])
    out[:len(picked)] = picked
    return out


def masked_rows(rng, longest):
    """Rows of at most `longest` scores whose 512th best is a mask, or next to one: (lengths, bits)."""
    lengths, rows = [], []
    for length in sorted({513, 520, 543, 640, 1000, 1023, 1024, longest - 1, longest} | ({1030, longest // 2 + 1} if longest > 1024 else set())):
        for masks in (1, 2, 10, 20, 31, 32, 33, 40):
            kind = len(rows)
            values = rng.normal(size=longest).astype(np.float32) - 4
            values[0] = HIGHEST[kind % len(HIGHEST)]
            values[1:] = np.minimum(values[1:], values[0])
            bits = values.view(np.uint32)
            high = 512 - int(rng.integers(0, masks + 1))    # scores above the masks: the threshold is a mask, or the lowest of these
            if length - masks > high:                       # others far below the masks
                bits[high:length - masks] = 0xFFFFFFF0 - np.arange(length - masks - high) if MASKS[kind % 4] < 0xFFFFFFFF else MASKS[0]
            bits[max(length - masks, 1):length] = MASKS[kind % 4]
            bits[:length] = rng.permutation(bits[:length])
            rows.append(bits)
            lengths.append(length)
    return lengths, np.array(rows)


@pytest.mark.parametrize("rows,longest", [(2000, 1024), (300, 1024), (280, 1030), (100, 2048), (101, 4096)])  # 128, 256, half of 512, 512 threads, and 1024 by the widths below
def test_masks_at_the_threshold_of_rows_that_are_listed_whole(select, rows, longest):
    lengths, bits = masked_rows(np.random.default_rng(rows), longest)
    width = {4096: 140000, 1030: 33000}.get(longest, longest + 4)
    wide = np.zeros((len(bits), width), dtype=np.uint32)
    wide[:, :longest] = bits
    picked = select(rows, lengths, wide)
    for row, length in enumerate(lengths):
        assert np.array_equal(picked[row], best(bits[row, :length])), (row, length)


@pytest.mark.parametrize("rows,span", [(2000, 6000), (300, 6000), (280, 40000), (100, 9000), (101, 140000)])
def test_rows_that_are_sampled(select, rows, span):
    """The usual way, and the one by keys behind lists that are too long or too short."""
    rng = np.random.default_rng(span)
    scores = rng.normal(size=(8, span)).astype(np.float32)
    few = rng.choice(span, 400, replace=False)
    scores[1] = 0.25
    scores[2] = np.where(np.isin(np.arange(span), few), scores[2], -np.inf)
    scores[3] = np.maximum(scores[3] - 2.9, 0)
    scores[4] = np.sort(scores[4])
    scores[5, 40:400] = 30
    bits = scores.view(np.uint32)
    bits[6, 600:] = 0xFFC00000
    bits[7, rng.choice(span, 900, replace=False)] = 0xFFFFFFFF
    lengths = [span - (row % 3) for row in range(len(bits))]
    picked = select(rows, lengths, bits)
    for row, length in enumerate(lengths):
        assert np.array_equal(picked[row], best(bits[row, :length])), row
