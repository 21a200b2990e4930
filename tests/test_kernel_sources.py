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


def test_a_rescale_tells_the_end_of_the_products_before_it_from_earlier_ones():
    """A wait by parity passes on any phase that is not the present one, so whoever waits for the end of PV c - 1 has to know that the
    barrier's phase before that has ended. Arrivals of different commits come in no particular order: known is what somebody
    on the way to chunk c has waited for on the same barrier."""
    source = (CSRC / "sparse_mla_tcgen05.cuh").read_text()
    stages = int(re.search(r"constexpr int kStages = (\d+);", source).group(1))

    def barrier(expression, **names):  # (name, number) of "kName" or "kName0 + number"
        name, _, number = expression.partition("0 + ")
        return name, eval(number or "0", {"kStages": stages}, names)

    rescale = source[source.index("const float o_alpha = "):]
    waited, parity = re.search(r"warp_wait\(sm\.bar\((.+)\), (.+), abort_flag\)", rescale).groups()
    issue = source[source.index("void issue_pv("):source.index("void qk_role(")]
    commits = re.findall(r"mma_commit\(sm\.bar\((.+?)\)\);", issue.split("kPvSteps, false>")[-1])
    role = source[source.index("void pv_role("):source.index("void softmax_role(")]
    commits += re.findall(r"\n      mma_commit\(sm\.bar\((.+?)\)\);", role)
    producers = source[source.index("void producer_role("):source.index("void qk_role(")]
    gathered_behind = re.findall(r"use > 0 && !warp_wait\(sm\.bar\((.+?)\), \(use - 1\) & 1, abort_flag", producers)

    for chunk in range(1, 40):
        phase = eval(parity.replace("/", "//"), {"kStages": stages}, {"chunk_count": chunk})
        wanted = barrier(waited, chunk_count=chunk)
        ends = [k for k in range(chunk) if any(barrier(c, stage=k % stages, p_tile=k & 1) == wanted for c in commits)]
        assert ends and ends[-1] == chunk - 1, (chunk, wanted)
        # the producers brought tile k into its stage behind the end of PV k - kStages, and tiles 0 .. c have been multiplied
        known = [k - stages for k in range(stages, chunk) if any(barrier(b, stage=k % stages) == wanted for b in gathered_behind)]
        for phases in range(len(set(known) & set(ends)), len(ends)):
            assert phases & 1 == phase, (chunk, phases)  # waits
        assert len(ends) & 1 != phase  # passes


def test_slots_are_resolved_by_one_routine():
    """The rule from slot to row stands once beside the tcgen05 kernels, and all forms of resolving a token run it."""
    source = (CSRC / "sparse_mla_tcgen05.cuh").read_text()
    assert source.count("report(p, kStatusBadPage") == 1
    assert "kStatusBadPage" not in (CSRC / "sparse_mla_team.cuh").read_text()


@pytest.mark.parametrize("name", ["sparse_mla_tcgen05.cuh", "sparse_mla_team.cuh"])
def test_issuing_threads_are_elected(name):
    """A role that issues products runs in the thread that `elect.sync` chose: behind a comparison of the thread index calls of few
    tokens take a seventh longer."""
    kernel = (CSRC / name).read_text().split("__global__ void __launch_bounds__")[-1]
    calls = re.findall(r"(.*\b(?:qk_role|pv_role|team_qk|team_pv)<kFormat>)\(", kernel)
    assert [call.split()[:2] for call in calls] == [["if", "(elect_one())"]] * 2


@pytest.mark.parametrize("name", ["sparse_mla_tcgen05.cuh", "sparse_mla_team.cuh"])
def test_a_wait_that_gave_up_is_looked_for_behind_a_barrier_of_the_whole_block(name):
    """Any role's last wait can give up after other warps have left theirs; the softmax warps of a cluster arrive at its last barrier
    before such a wait. So the flag is read behind a barrier that every warp comes to with nothing left to wait for."""
    kernel = (CSRC / name).read_text().split("__global__ void __launch_bounds__")[-1]
    roles_end = max(kernel.index("producer_role(p") if "producer_role(p" in kernel else 0, kernel.find("team_slices(p"))
    behind = kernel[roles_end:kernel.index("report(p, kStatusWaitExpired")]
    assert behind.rfind("__syncthreads();") > behind.rfind("cluster_wait();")
