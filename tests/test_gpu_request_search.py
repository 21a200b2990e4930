"""The resolver's request search at the edges of its 32-wide steps: the exported index set against the
oracle, with empty requests first, last and in runs."""

import numpy as np
import pytest

from oracle import sparse_mla_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("requests", [1, 2, 31, 32, 33, 63, 64, 65, 1023, 1025])
def test_search_finds_the_request_of_every_token(requests):
    import torch

    from ascendflow_b200 import ops

    rng = np.random.default_rng(requests)
    counts = rng.integers(0, 3, requests)
    counts[rng.random(requests) < 0.3] = 0
    counts[requests // 2] = 2
    tokens, pages = int(counts.sum()), 4
    lengths = np.maximum(counts, rng.integers(1, pages * 128 + 1, requests)).astype(np.int32)
    policy = O.make_policy(requests, tokens, ratio=2, max_seq=pages * 128, blocks=requests * pages)
    indices = np.full((tokens, 1, 512), -1, dtype=np.int32)
    for token in range(tokens):
        take = int(rng.integers(0, 200))
        indices[token, 0, :take] = np.sort(rng.choice(pages * 64, take, replace=False))
    table = rng.permutation(requests * pages).reshape(requests, pages).astype(np.int32)
    data = {
        "cmp_sparse_indices": indices, "ori_block_table": table, "cmp_block_table": table[::-1].copy(),
        "cu_seqlens_q": np.concatenate([[0], np.cumsum(counts)]).astype(np.int32), "seqused_ori_kv": lengths,
        "seqused_cmp_kv": lengths // 2, "cmp_residual_kv": lengths % 2,
        "ori_topk_length": rng.integers(0, 140, (tokens, 1)).astype(np.int32),
    }
    names = ("cmp_sparse_indices", "ori_block_table", "cmp_block_table", "cu_seqlens_q", "seqused_ori_kv", "seqused_cmp_kv",
             "cmp_residual_kv", "ori_topk_length")
    resolved = ops.resolve_rows(*(torch.from_numpy(np.ascontiguousarray(data[n])).cuda() for n in names),
                                ori_blocks=requests * pages, cmp_blocks=requests * pages, cmp_page=64)
    assert np.array_equal(resolved.cpu().numpy(), O.resolve_rows(data, policy))
