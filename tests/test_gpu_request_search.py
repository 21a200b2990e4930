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


@pytest.mark.parametrize("requests", [1, 2, 31, 32, 33, 64, 1025])
def test_append_and_selection_find_the_request_of_every_token(requests):
    """The cache append, and the selection of few rows, whose lanes load a request's scalars with the probe."""
    import torch

    from ascendflow_b200 import neighbours

    rng = np.random.default_rng(requests)
    counts = np.zeros(requests, dtype=np.int64)
    counts[rng.choice(requests, min(requests, 40), replace=False)] = rng.integers(1, 3, min(requests, 40))
    tokens, pages = int(counts.sum()), 8
    cu = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    lengths = np.maximum(counts, rng.integers(1, pages * 128 + 1, requests)).astype(np.int32)
    table = rng.permutation(requests * pages).reshape(requests, pages).astype(np.int32)
    used = int(table.max()) + 1
    cache, rows = np.zeros((used, 128, 1, 512), dtype=np.int16), rng.integers(-32768, 32768, (tokens, 512)).astype(np.int16)
    on_gpu = lambda array: torch.from_numpy(np.ascontiguousarray(array)).cuda()
    device_cache = on_gpu(cache).view(torch.bfloat16)
    status = neighbours.cache_append(on_gpu(rows).view(torch.bfloat16), device_cache, on_gpu(table), on_gpu(cu), on_gpu(lengths))
    assert tuple(status) == (0,) * 8
    assert np.array_equal(device_cache.view(torch.int16).cpu().numpy(), O.append_rows(cache, rows, table, cu, lengths))

    data = {"cu_seqlens_q": cu, "seqused_ori_kv": lengths, "seqused_cmp_kv": lengths, "cmp_residual_kv": np.zeros(requests, dtype=np.int32)}
    policy = O.make_policy(requests, tokens, ratio=1, max_seq=pages * 128, blocks=8)
    scores = rng.normal(size=(tokens, pages * 128)).astype(np.float32)
    selected = neighbours.topk_indices(on_gpu(scores), on_gpu(cu), on_gpu(lengths), on_gpu(data["cmp_residual_kv"]), ratio=1)
    assert np.array_equal(selected.cpu().numpy(), O.select_topk_indices(scores, data, policy))


@pytest.mark.parametrize("requests", [1, 2, 33, 1100])
def test_tokens_in_front_of_the_first_request_count_to_it(requests):
    """`cu_seqlens_q` need not start at 0: the binary search of the search's contract ends at request 0."""
    import torch

    from ascendflow_b200 import neighbours, ops

    front, length, pages = 5, 300, 4
    tokens = front + requests
    cu = front + np.arange(requests + 1, dtype=np.int32)
    table = np.random.default_rng(1).permutation(requests * pages).reshape(requests, pages).astype(np.int32)
    of = np.maximum(0, np.arange(tokens) - front)                       # request of every token
    position = length - 1 + np.minimum(0, np.arange(tokens) - front)    # last row it sees, its own
    on_gpu = lambda array: torch.from_numpy(np.ascontiguousarray(array)).cuda()  # noqa: E731
    lengths, zeros = np.full(requests, length, dtype=np.int32), np.zeros(requests, dtype=np.int32)

    none = np.full((tokens, 1, 512), -1, dtype=np.int32)
    resolved = ops.resolve_rows(*map(on_gpu, (none, table, table, cu, lengths, lengths, zeros, np.zeros((tokens, 1), dtype=np.int32))),
                                ori_blocks=requests * pages, cmp_blocks=requests * pages, cmp_page=128).cpu().numpy()
    window = position[:, None] - 127 + np.arange(128)
    assert np.array_equal(resolved[:, :128], table[of[:, None], window // 128] * 128 + window % 128)

    rows = np.random.default_rng(2).integers(-32768, 32768, (tokens, 512)).astype(np.int16)
    cache = torch.zeros((requests * pages, 128, 1, 512), dtype=torch.bfloat16, device="cuda")
    status = neighbours.cache_append(on_gpu(rows).view(torch.bfloat16), cache, on_gpu(table), on_gpu(cu), on_gpu(lengths))
    assert tuple(status) == (0,) * 8
    written = cache.view(-1, 512).view(torch.int16).cpu().numpy()
    assert np.array_equal(written[table[of, position // 128] * 128 + position % 128], rows)

    scores = np.random.default_rng(3).normal(size=(tokens, 512)).astype(np.float32)
    selected = neighbours.topk_indices(on_gpu(scores), on_gpu(cu), on_gpu(lengths), on_gpu(zeros), ratio=1).cpu().numpy()
    for token in range(tokens):
        assert np.array_equal(selected[token, 0], np.where(np.arange(512) <= position[token], np.arange(512), -1))
