"""Index lists that are not sorted and padded: the exported index set, which resolves every token in the form in which a
call of that many tokens gathers it (five warps for the first token of a block, one warp for the others), against the
oracle, and the output of the same call."""

import numpy as np
import pytest

from oracle import sparse_mla_oracle as O
from tests import support as S

pytestmark = pytest.mark.gpu

NAMES = ("cmp_sparse_indices", "ori_block_table", "cmp_block_table", "cu_seqlens_q", "seqused_ori_kv", "seqused_cmp_kv",
         "cmp_residual_kv", "ori_topk_length")
MAX_SEQ = 2048
KINDS = 9


def index_list(rng, kind, span):
    """512 entries below `span`, most in no order, with duplicates."""
    row = rng.integers(0, span, 512)
    if kind == 0:
        row = np.sort(row)
    elif kind <= 4:  # the list ends in a quarter of its own, valid entries behind
        row[(kind - 1) * 128 + rng.choice([0, 31, 32, 127, int(rng.integers(128))])] = -int(rng.integers(1, 1 << 31))
        row[rng.integers((kind - 1) * 128, 512, 3)] = -1
    elif kind == 5:
        row[0] = -1
    elif kind == 6:  # nothing else ends it
        row[511] = -1
    elif kind == 7:  # beyond any cutoff
        row[rng.integers(0, 512, 100)] = rng.integers(span, 1 << 31, 100)
    return row.astype(np.int32)


def call(tokens, requests, ratio, seed):
    rng = np.random.default_rng(seed)
    counts = np.full(requests, tokens // requests)
    counts[: tokens - counts.sum()] += 1
    pages = MAX_SEQ // 128
    lengths = np.maximum(counts, rng.integers(1, MAX_SEQ + 1, requests)).astype(np.int32)
    lengths[0] = MAX_SEQ
    policy = O.make_policy(requests, tokens, ratio=ratio, max_seq=MAX_SEQ)
    rows = [index_list(rng, token % KINDS, MAX_SEQ // ratio) for token in range(tokens)]
    data = {
        "cmp_sparse_indices": np.stack(rows)[:, None],
        "ori_block_table": rng.permutation(requests * pages).reshape(requests, pages).astype(np.int32),
        "cmp_block_table": rng.permutation(requests * pages).reshape(requests, pages).astype(np.int32),
        "cu_seqlens_q": np.concatenate([[0], np.cumsum(counts)]).astype(np.int32), "seqused_ori_kv": lengths,
        "seqused_cmp_kv": lengths // ratio, "cmp_residual_kv": lengths % ratio,
        "ori_topk_length": rng.choice([0, 0, 1, 70, 128], (tokens, 1)).astype(np.int32),
    }
    return data, policy


def tensors_of(data, policy, seed):
    import torch

    generator = torch.Generator(device="cuda")
    generator.manual_seed(seed)
    normal = lambda *shape: torch.randn(shape, dtype=torch.bfloat16, device="cuda", generator=generator)  # noqa: E731
    tensors = {name: torch.from_numpy(np.ascontiguousarray(value)).cuda() for name, value in data.items()}
    blocks = policy["ORI_BLOCKS"]
    tensors.update(q=normal(policy["T"], 64, 512), ori_kv=normal(blocks, 128, 1, 512),
                   cmp_kv=normal(blocks, 128 // policy["RATIO"], 1, 512), sinks=torch.linspace(-3, 3, 64, device="cuda"))
    tensors["attention_out"] = torch.full_like(tensors["q"], float("nan"))
    return tensors


def exported(tensors, policy):
    from ascendflow_b200 import ops

    return ops.resolve_rows(*(tensors[name] for name in NAMES), ori_blocks=policy["ORI_BLOCKS"],
                            cmp_blocks=policy["CMP_BLOCKS"], cmp_page=128 // policy["RATIO"]).cpu().numpy()


def call_sizes(ratios):
    """A cluster per token; a block per token; one more than blocks; groups of two and a rest."""
    return [(tokens, requests, ratio) for ratio in ratios
            for tokens, requests in ((1, 1), (9, 9), (18, 2), (40, 40), (148, 33), (149, 70), (1200, 7))]


@pytest.mark.parametrize("tokens,requests,ratio", call_sizes((1, 2)))
def test_lists_of_every_kind(tokens, requests, ratio):
    from ascendflow_b200 import ops

    data, policy = call(tokens, requests, ratio, tokens + ratio)
    tensors = tensors_of(data, policy, tokens)
    assert np.array_equal(exported(tensors, policy), O.resolve_rows(data, policy))
    assert ops.kernel().bind(*(tensors[name] for name in S.TENSOR_ORDER))().status()[0] == 0
    sample = sorted({*range(min(tokens, KINDS)), *range(max(0, tokens - KINDS), tokens)})
    actual = S.output_to_numpy(tensors["attention_out"], "bf16")
    assert np.isfinite(actual).all()
    S.assert_close(actual[sample], S.sampled_reference(tensors, data, policy, sample), "lists")


@pytest.mark.parametrize("table", ["ori_block_table", "cmp_block_table"])
@pytest.mark.parametrize("tokens,requests,ratio", call_sizes((2,)))
def test_bad_pages_are_masked_and_reported(tokens, requests, ratio, table):
    """Page numbers outside of the cache, below and above, and positions whose page the table does not list: host checks
    cannot see them, the kernel's own turn them into masked slots and a report."""
    import torch

    from ascendflow_b200 import ops

    data, policy = call(tokens, requests, ratio, tokens)
    rng = np.random.default_rng(tokens)
    data[table][rng.random(data[table].shape) < 0.2] = policy["ORI_BLOCKS"] + 5
    data[table][rng.random(data[table].shape) < 0.2] = -3
    data[table][0, -1] = policy["ORI_BLOCKS"]  # the first request is the longest: someone reads it
    whole = O.resolve_rows(data, policy)
    expected = whole.copy()
    limits = np.array([policy["ORI_BLOCKS"] * 128] * 128 + [policy["CMP_BLOCKS"] * 128 // ratio] * 512)
    expected[(whole < 0) | (whole >= limits)] = -1
    tensors = tensors_of(data, policy, tokens)
    assert np.array_equal(exported(tensors, policy), expected)
    status = ops.kernel().bind(*(tensors[name] for name in S.TENSOR_ORDER))().status()
    assert status[0] == 1 and (expected[status[1]] != whole[status[1]]).any()
    assert bool(torch.isfinite(tensors["attention_out"]).all())
    # The table one page short: what lies behind is masked too.
    for name in ("ori_block_table", "cmp_block_table"):
        tensors[name] = tensors[name][:, :-1].contiguous()
    pages = np.full_like(whole, -1)
    geometry = O.token_geometry(data, policy)
    pages[:, :128] = ((geometry["right"] - geometry["visible"])[:, None] + np.arange(128)) // 128
    pages[:, 128:] = data["cmp_sparse_indices"][:, 0] // (128 // ratio)
    expected[pages == MAX_SEQ // 128 - 1] = -1
    assert np.array_equal(exported(tensors, policy), expected)
