"""The steps next to the operator: top-k index selection and cache append.

CPU: the oracle's definitions on hand-sized cases, and that what the selection produces is what
the operator's row selection accepts in full. GPU: the CUDA kernels against the oracle, bit for
bit (int32 indices, cache bytes), through the C ABI.
"""

import numpy as np
import pytest

from oracle import sparse_mla_oracle as O


def small(b=2, t=6, lengths=(40, 9), ratio=2):
    policy = O.make_policy(b, t, h=2, d=8, page=8, ratio=ratio, max_seq=64, window=4, topk=4, blocks=16)
    counts = O.query_counts(policy)
    lengths = np.asarray(lengths, dtype=np.int32)
    data = {
        "cu_seqlens_q": np.concatenate([[0], np.cumsum(counts)]).astype(np.int32),
        "seqused_ori_kv": lengths,
        "seqused_cmp_kv": (lengths // ratio).astype(np.int32),
        "cmp_residual_kv": (lengths % ratio).astype(np.int32),
    }
    return policy, data


def test_selection_takes_the_highest_scores_lowest_index_first_on_ties():
    policy, data = small()
    scores = np.zeros((6, 32), dtype=np.float32)
    scores[0, [3, 7, 11, 15, 16]] = [5, 4, 4, 4, 4]     # four of five: the tie at 4 is cut by index
    picked = O.select_topk_indices(scores, data, policy)
    geometry = O.token_geometry(dict(data, ori_topk_length=np.zeros((6, 1), np.int32)), policy)
    assert picked[0, 0].tolist() == [3, 7, 11, 15]
    # request 1 holds 9 rows and 3 queries: token 3 sees (9 - 3 + 0 + 1) // 2 = 3 compressed rows
    assert geometry["cutoff"][3] == 3 and picked[3, 0].tolist() == [0, 1, 2, -1]
    # all scores equal: the first TOPK visible rows
    assert picked[1, 0].tolist() == [0, 1, 2, 3]


def test_selection_is_accepted_in_full_by_the_operators_row_selection():
    rng = np.random.default_rng(5)
    policy = O.make_policy(3, 30, max_seq=4096, blocks=96)
    data = O.validation_inputs(policy, "mixed")
    scores = rng.normal(size=(30, 2048)).astype(np.float32)
    data["cmp_sparse_indices"] = O.select_topk_indices(scores, data, policy)
    resolved = O.resolve_rows(data, policy)
    geometry = O.token_geometry(data, policy)
    for token in range(30):
        listed = data["cmp_sparse_indices"][token, 0]
        live = listed[listed >= 0]
        assert len(live) == min(512, geometry["available"][token], geometry["cutoff"][token])
        assert (np.diff(live) > 0).all()
        assert (resolved[token, 128:128 + len(live)] >= 0).all() and (resolved[token, 128 + len(live):] < 0).all()


def test_append_puts_rows_where_the_window_looks_for_them():
    policy, data = small()
    rng = np.random.default_rng(2)
    cache = rng.normal(size=(16, 8, 1, 8)).astype(np.float32)
    table = np.stack([rng.permutation(8), rng.permutation(8) + 8]).astype(np.int32)
    new = rng.normal(size=(6, 8)).astype(np.float32)
    after = O.append_rows(cache, new, table, data["cu_seqlens_q"], data["seqused_ori_kv"])
    # token 5 is the last of request 1 (length 9): position 8 = page table[1][1], row 0
    assert np.array_equal(after[table[1, 1], 0, 0], new[5])
    assert np.array_equal(after[table[0, 4], 7, 0], new[2])          # request 0: positions 37, 38, 39
    changed = (after != cache).any(axis=(2, 3)).sum()
    assert changed == 6


@pytest.mark.gpu
@pytest.mark.parametrize("ratio,seed", [(2, 0), (2, 1), (1, 2)])
def test_gpu_selection_matches_the_oracle_bit_for_bit(ratio, seed):
    import torch

    from ascendflow_b200 import neighbours

    rng = np.random.default_rng(40 + seed)
    lens = [int(v) for v in rng.integers(0, 40, 5)]
    lens[0] = max(lens[0], 3)
    policy = O.make_policy(len(lens), sum(lens), ratio=ratio, max_seq=8192, blocks=8)
    lengths = np.array([int(rng.integers(max(n, 1), 8193)) for n in lens], dtype=np.int32)
    lengths[1] = max(lens[1], 1)                      # a cache that holds only its queries
    data = {
        "cu_seqlens_q": np.concatenate([[0], np.cumsum(lens)]).astype(np.int32),
        "seqused_ori_kv": lengths,
        "seqused_cmp_kv": (lengths // ratio).astype(np.int32),
        "cmp_residual_kv": (lengths % ratio).astype(np.int32),
    }
    span = 8192 // ratio
    scores = rng.normal(size=(sum(lens), span)).astype(np.float32)
    scores[::3] = np.round(scores[::3] * 2) / 2       # plenty of exact ties
    scores[5] = 1.25                                  # one token with nothing but ties
    expected = O.select_topk_indices(scores, data, policy)
    device = {k: torch.from_numpy(v).cuda() for k, v in data.items()}
    actual = neighbours.topk_indices(torch.from_numpy(scores).cuda(), device["cu_seqlens_q"], device["seqused_cmp_kv"],
                                     device["cmp_residual_kv"], ratio=ratio)
    assert np.array_equal(actual.cpu().numpy(), expected)


@pytest.mark.gpu
@pytest.mark.parametrize("max_seq,ratio", [(131072, 2), (32768, 2), (131072, 1), (262144, 2)])
def test_gpu_selection_over_long_rows(max_seq, ratio):
    """Decode-sized rows, selected from one read, and one longer than a window of winners. Continuous scores,
    heavy ties, one row of nothing but ties (more of them than the list holds), one of negative values."""
    import torch

    from ascendflow_b200 import neighbours

    rng = np.random.default_rng(max_seq // 1024 + ratio)
    lens = [2, 1, 3, 2]
    span = max_seq // ratio
    policy = O.make_policy(len(lens), sum(lens), ratio=ratio, max_seq=max_seq, blocks=8)
    lengths = np.array([max_seq, max_seq - 5, 4100, 700], dtype=np.int32)   # long, long, short, under TopK
    data = {
        "cu_seqlens_q": np.concatenate([[0], np.cumsum(lens)]).astype(np.int32),
        "seqused_ori_kv": lengths,
        "seqused_cmp_kv": (lengths // ratio).astype(np.int32),
        "cmp_residual_kv": (lengths % ratio).astype(np.int32),
    }
    scores = rng.normal(size=(sum(lens), span)).astype(np.float32)
    scores[1] = np.round(scores[1] * 4) / 4           # a few dozen distinct values: long runs of ties
    scores[2] = -3.5                                  # nothing but ties
    scores[3] = -np.abs(scores[3])                    # negative keys only
    scores[4, ::7] = np.float32(2.0)                  # a plateau that the threshold falls into
    expected = O.select_topk_indices(scores, data, policy)
    device = {k: torch.from_numpy(v).cuda() for k, v in data.items()}
    actual = neighbours.topk_indices(torch.from_numpy(scores).cuda(), device["cu_seqlens_q"], device["seqused_cmp_kv"],
                                     device["cmp_residual_kv"], ratio=ratio)
    assert np.array_equal(actual.cpu().numpy(), expected)


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,visible", [
    # 256-thread blocks: TopK, listed whole (1024), the list (2560), one step of the stream (4096), the sample's
    # sizes, the window of winners (65536), each with its neighbours
    (320, (1, 4, 511, 512, 513, 1024, 1025, 2559, 2560, 2561, 4095, 4097, 16383, 32769, 65535, 65536, 65537, 70001)),
    # 512-thread blocks: listed whole (2048), the list (4096), one step (8192), the longest
    (19, (512, 513, 2047, 2048, 2049, 4096, 4097, 8191, 8192, 8193, 16384, 16385, 131071, 131072, 65537)),
    # 1024-thread blocks: listed whole (4096), the list (8192), one step (16384), more than a window of winners
    (7, (4096, 4097, 8193, 16385, 131073, 200001, 150000)),
    # 128-thread blocks, ten per SM (rows of at most 10240 scores): the list and one step (2048)
    (1900, (511, 512, 513, 2047, 2048, 2049, 3000, 4095, 4097, 6143, 8191, 8192)),
    # 128-thread blocks, eight per SM: the list (2048), one step (4096), the window of winners (32768), the longest
    (1800, (511, 512, 513, 2047, 2048, 2049, 3000, 4095, 4097, 8191, 16385, 32767, 32768)),
])
def test_gpu_selection_at_the_edges_of_its_blocks(tokens, visible):
    """One token per request, every row length in turn; continuous, 8-bit-mantissa, offset,
    clustered and few-valued scores in turn (what a sample of the row says about it differs)."""
    import torch

    from ascendflow_b200 import neighbours

    rng = np.random.default_rng(tokens)
    policy = O.make_policy(tokens, tokens, ratio=1, max_seq=-(-max(max(visible), 131072) // 128) * 128, blocks=8)
    lengths = np.array([visible[i % len(visible)] for i in range(tokens)], dtype=np.int32)
    data = {
        "cu_seqlens_q": np.arange(tokens + 1, dtype=np.int32),
        "seqused_ori_kv": lengths, "seqused_cmp_kv": lengths,
        "cmp_residual_kv": np.zeros(tokens, dtype=np.int32),
    }
    span = -(-max(visible) // 4) * 4
    scores = rng.normal(size=(tokens, span)).astype(np.float32)
    for token in range(tokens):
        kind = (token // len(visible) + token) % 5
        if kind == 1:
            scores[token] = (scores[token].view(np.uint32) & 0xFFFF0000).view(np.float32)
        elif kind == 2:
            scores[token] += 1000.0
        elif kind == 3:  # the winners side by side, between the places a sample looks at
            first = int(rng.integers(0, max(1, lengths[token] - 600)))
            scores[token, first:first + 600] += 50.0
        elif kind == 4:  # hundreds of equal scores at the threshold: the position decides
            # (+ 0.0: no negative zeros, which the kernel's keys have always put below zero and the oracle ties with it)
            scores[token] = np.round(scores[token] * 8) / 8 + np.float32(0.0)
    expected = O.select_topk_indices(scores, data, policy)
    device = {k: torch.from_numpy(v).cuda() for k, v in data.items()}
    actual = neighbours.topk_indices(torch.from_numpy(scores).cuda(), device["cu_seqlens_q"], device["seqused_cmp_kv"],
                                     device["cmp_residual_kv"], ratio=1)
    assert np.array_equal(actual.cpu().numpy(), expected)


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,visible", [
    (1790, [16384, 16383, 513, 9000]), (1790, [16388, 16384, 700]),   # many rows, one window of winners or more
    (1790, [8192, 1025, 8191]), (148, [16388, 512, 20000]), (148, [16384, 2049]),  # a row per SM, either number of loads
    (149, [16388, 1]), (149, [16384, 16383, 2561]), (20, [131072, 16388, 65537]),
    (2368, [16000, 9000, 12289]), (2369, [16384, 10241]), (1800, [10240, 700]), (1800, [10244, 10241, 10240]),  # waves of eight and of ten blocks
    (296, [32772, 32768, 700]), (296, [32768, 4097]), (297, [32772, 20000]),  # two rows per SM
    (149, [40000, 16384, 16385, 16383, 1025, 1024, 513, 512]), (296, [65536, 16385, 2560, 2561, 1024, 1]),  # all of a block or half of it
    (297, [98308, 98304, 1025]), (297, [98304, 30000]), (300, [131072, 98304, 98305, 40000, 8192, 1025]),  # the larger sample, of long rows
    (297, [16388, 16384, 513]), (297, [24576, 24575, 16385, 700]), (297, [24580, 24576]),  # bitmaps of 16, 24 and 64 K
    (444, [32768, 24577]), (446, [24580, 24577, 1025]), (446, [32768, 32767, 30001, 2561]), (446, [32772, 32768]),
    (446, [49152, 49151, 40001]), (446, [49156, 49152]), (444, [49152]),  # or 32 and 48 K
    (296, [131076, 513]), (297, [131076, 700]),  # scores copied or listed with their positions
    (148, [24576, 24575, 4096]), (148, [24580, 24576, 24577, 24575, 2049, 700, 512]),  # the row's own length chooses it
])
def test_gpu_selection_at_the_lines_between_its_kernels(tokens, visible):
    test_gpu_selection_at_the_edges_of_its_blocks(tokens, visible)


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,visible", [
    (1800, [1024, 1023, 1025, 896, 897, 641, 640, 513]),  # 128 threads: lists that fill their last round, all but fill it, begin one
    (300, [1024, 1023, 1025, 769, 768, 513]),             # 256
    (140, [2048, 2047, 2049, 1537, 1536, 1024, 513]),     # 512
])
def test_gpu_selection_from_lists_that_end_on_a_round_of_their_block(tokens, visible):
    """Rows as short as these are listed in full: the list is as long as the row."""
    test_gpu_selection_at_the_edges_of_its_blocks(tokens, visible)


@pytest.mark.gpu
@pytest.mark.parametrize("tokens", [7, 140, 300, 1800])  # 512 threads twice, 256, 128
def test_gpu_selection_with_every_number_of_scores_at_its_threshold(tokens):
    """One to 34 equal scores, the threshold among them: up to 32 are ranked by one warp, eight at a time or one by one."""
    import torch

    from ascendflow_b200 import neighbours

    rng = np.random.default_rng(tokens)
    span = 1000
    policy = O.make_policy(tokens, tokens, ratio=1, max_seq=1024, blocks=8)
    lengths = np.full(tokens, span, dtype=np.int32)
    data = {
        "cu_seqlens_q": np.arange(tokens + 1, dtype=np.int32),
        "seqused_ori_kv": lengths, "seqused_cmp_kv": lengths,
        "cmp_residual_kv": np.zeros(tokens, dtype=np.int32),
    }
    scores = np.empty((tokens, span), dtype=np.float32)
    for token in range(tokens):
        equal = 1 + token % 34 if tokens > 34 else (1, 8, 9, 16, 17, 32, 33)[token]
        inside = int(rng.integers(1, equal + 1))                 # of them win
        better = 512 - inside
        row = np.concatenate([rng.uniform(2e4, 4e4, better), np.full(equal, 1e4), rng.uniform(0, 10, span - better - equal)])
        scores[token] = rng.permutation(row)
    expected = O.select_topk_indices(scores, data, policy)
    device = {k: torch.from_numpy(v).cuda() for k, v in data.items()}
    actual = neighbours.topk_indices(torch.from_numpy(scores).cuda(), device["cu_seqlens_q"], device["seqused_cmp_kv"],
                                     device["cmp_residual_kv"], ratio=1)
    assert np.array_equal(actual.cpu().numpy(), expected)


@pytest.mark.gpu
def test_gpu_selection_feeds_the_attention_call():
    """Scores -> indices on the device -> attention, against the oracle fed with the oracle's selection."""
    import torch

    from ascendflow_b200 import neighbours, ops
    from tests import support as S

    policy = O.make_policy(4, 16, max_seq=4096, blocks=128)
    data = O.validation_inputs(policy, "mixed")
    rng = np.random.default_rng(9)
    scores = rng.normal(size=(16, 2048)).astype(np.float32)
    data["cmp_sparse_indices"] = O.select_topk_indices(scores, data, policy)
    tensors, _ = S.to_device(data, policy)
    tensors["cmp_sparse_indices"] = neighbours.topk_indices(
        torch.from_numpy(scores).cuda(), tensors["cu_seqlens_q"], tensors["seqused_cmp_kv"], tensors["cmp_residual_kv"])
    assert np.array_equal(tensors["cmp_sparse_indices"].cpu().numpy(), data["cmp_sparse_indices"])
    ops.sparse_mla(*(tensors[name] for name in S.TENSOR_ORDER))
    S.assert_close(S.output_to_numpy(tensors["attention_out"], "bf16"), O.reference_fp32_from_data(data, policy), "selected on the device")


@pytest.mark.gpu
def test_gpu_append_matches_the_oracle_byte_for_byte():
    import torch

    from ascendflow_b200 import neighbours

    rng = np.random.default_rng(77)
    lens = [6, 0, 130, 1]
    lengths = np.array([700, 5, 130, 4096], dtype=np.int32)
    pages, blocks = 32, 4 * 32
    table = np.stack([rng.permutation(pages) + b * pages for b in range(4)]).astype(np.int32)
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cache = rng.integers(0, 1 << 16, size=(blocks, 128, 1, 512), dtype=np.uint16)
    new = rng.integers(0, 1 << 16, size=(sum(lens), 512), dtype=np.uint16)
    expected = O.append_rows(cache, new, table, cu, lengths)
    as_bf16 = lambda a: torch.from_numpy(a.view(np.int16)).cuda().view(torch.bfloat16)
    device_cache = as_bf16(cache)
    status = neighbours.cache_append(as_bf16(new), device_cache, torch.from_numpy(table).cuda(),
                                     torch.from_numpy(cu).cuda(), torch.from_numpy(lengths).cuda())
    assert status[0] == 0
    assert np.array_equal(device_cache.view(torch.int16).cpu().numpy().view(np.uint16), expected)
    # a length beyond the table: reported, nothing written there, the context stays usable
    bad = lengths.copy()
    bad[3] = pages * 128 + 1
    status = neighbours.cache_append(as_bf16(new), device_cache, torch.from_numpy(table).cuda(),
                                     torch.from_numpy(cu).cuda(), torch.from_numpy(bad).cuda())
    assert status[0] == 1 and status[1] == sum(lens) - 1


def selection_steps(source):
    """The type and the step of the loop over the windows of winners, from the kernel's source."""
    import re

    kind, step = re.search(r"for \((\w+) window = 0; window < \w+; window \+= (\w+)\)", source).groups()
    return kind, {"kWindow": 65536}[step]


def test_windows_of_winners_end_on_the_longest_row():
    """The last window of the longest accepted row starts below 2^31 and ends above: the position behind it must
    not come out negative (the loop would not end)."""
    from pathlib import Path

    kind, step = selection_steps((Path(__file__).resolve().parents[1] / "ascendflow_b200/csrc/sparse_mla_neighbours.cu").read_text())
    longest = 2**31 - 1 - 8192
    behind = (longest - 1) // step * step + step
    wrapped = behind - 2**32 if kind == "int" and behind >= 2**31 else behind % 2**32
    assert wrapped >= longest


@pytest.mark.gpu
def test_gpu_selection_over_the_longest_row():
    """2^31 - 8196 scores (8.6 GB). The sampled head of the row holds high scores, so that the list is short and
    its winners are put in order window by window, up to the row's end."""
    import torch

    from ascendflow_b200 import neighbours

    span = 2**31 - 1 - 8192 - 3
    scores = torch.empty((1, span), dtype=torch.float32, device="cuda").normal_()
    generator = torch.Generator(device="cuda")
    generator.manual_seed(3)
    for first, count in ((0, 900), (span // 2 + 5000, 300), (span - 70000, 300), (span - 300, 300)):
        scores[0, first:first + count] = 100 + torch.rand(count, device="cuda", generator=generator)
    i32 = lambda *values: torch.tensor(values, dtype=torch.int32, device="cuda")  # noqa: E731
    actual = neighbours.topk_indices(scores, i32(0, 1), i32(span), i32(0), ratio=1)[0, 0].long()
    places = torch.cat([torch.arange(first, first + count) for first, count in ((0, 900), (span // 2 + 5000, 300), (span - 70000, 300), (span - 300, 300))]).cuda()
    order = torch.argsort(scores[0, places], descending=True, stable=True)   # ties: the lower index
    assert torch.equal(actual, places[order[:512]].sort().values)


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,span", [(1800, 14336), (1800, 4096), (320, 65536), (320, 14336), (19, 16384), (19, 40000), (7, 150000)])  # 128 (twice), 256, 512, 1024 threads
def test_gpu_selection_orders_what_is_not_finite_by_its_bits(tokens, span):
    """NaNs above and below the infinities by their sign, masks of -inf and of the lowest finite value, more and
    fewer of them than are selected."""
    import torch

    from ascendflow_b200 import neighbours

    rng = np.random.default_rng(span)
    scores = rng.normal(size=(tokens, span)).astype(np.float32)
    bits = scores.view(np.uint32)
    for token in range(tokens):
        few, many = rng.choice(span, 300, replace=False), rng.choice(span, 2000, replace=False)
        kind = token % 10
        if kind == 9:                                 # NaNs with a sign next to the floor, in order of their keys
            scores[token] = np.finfo(np.float32).min
            bits[token, many] = 0xFF800001
            scores[token, few] = rng.normal(size=300) * 1e37
        elif kind == 0:
            bits[token, many] = 0xFFC00000            # more NaNs with a sign than the list has room for beside the winners
        elif kind == 1:                               # few winners above the sample's floor, NaNs with a sign beside them
            first = int(rng.integers(0, span - 700))
            scores[token, first:first + 400] += 50.0
            bits[token, many[:700]] = 0xFFFFFFFF
        elif kind == 2:
            bits[token, few] = 0x7FC00000
            bits[token, many] = 0xFFC00001
        elif kind == 3:
            bits[token, many] = 0x7F800001 + np.arange(2000, dtype=np.uint32) % 7
        elif kind == 4:                               # nearly everything is masked: the threshold is a mask
            scores[token, np.setdiff1d(np.arange(span), few)] = -np.inf
        elif kind == 5:
            scores[token, np.setdiff1d(np.arange(span), many)] = np.finfo(np.float32).min
        elif kind == 6:
            scores[token] = -np.inf
            bits[token, few] = 0xFFC00000
        elif kind == 7:
            bits[token] = 0xFFC00000
            scores[token, many[:600]] = 1.0
        else:
            scores[token, many] = np.inf
    device = lambda array: torch.from_numpy(np.ascontiguousarray(array)).cuda()  # noqa: E731
    lengths = np.full(tokens, span, dtype=np.int32)
    actual = neighbours.topk_indices(device(scores), device(np.arange(tokens + 1, dtype=np.int32)), device(lengths),
                                     device(np.zeros(tokens, dtype=np.int32)), ratio=1).cpu().numpy()[:, 0]
    for token in range(tokens):
        key = np.where(bits[token] >> 31, ~bits[token], bits[token] | 0x80000000)
        threshold = np.sort(key)[-512]
        above, equal = np.flatnonzero(key > threshold), np.flatnonzero(key == threshold)
        assert np.array_equal(actual[token], np.sort(np.concatenate([above, equal[:512 - len(above)]])))


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,longest,width", [(1800, 1024, 1024), (320, 1024, 1024), (140, 2048, 2048), (280, 2048, 40000), (140, 4096, 140000)])  # 128, 256, 512 (twice), 1024 threads
def test_gpu_selection_with_masks_at_the_threshold_of_rows_that_are_listed_whole(tokens, longest, width):
    """Few masks, or NaNs with a sign, among which the threshold lies: the lowest bins, which reach down to the lowest key."""
    import torch

    from ascendflow_b200 import neighbours
    from tests.test_select_block import best, masked_rows

    lengths, bits = masked_rows(np.random.default_rng(tokens), longest)
    lengths = np.resize(np.array(lengths, dtype=np.int32), tokens)
    rows = np.full((tokens, width), 0xFFFFFFFF, dtype=np.uint32)
    rows[:, :longest] = bits[np.arange(tokens) % len(bits)]
    device = lambda array: torch.from_numpy(np.ascontiguousarray(array)).cuda()  # noqa: E731
    actual = neighbours.topk_indices(device(rows.view(np.float32)), device(np.arange(tokens + 1, dtype=np.int32)), device(lengths),
                                     device(np.zeros(tokens, dtype=np.int32)), ratio=1).cpu().numpy()[:, 0]
    for token in range(tokens):
        assert np.array_equal(actual[token], best(rows[token, :lengths[token]])), (token, lengths[token])


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,span", [(1800, 14336), (1800, 4096), (320, 65536), (320, 14336), (19, 16384), (19, 40000), (7, 150000)])  # as above
def test_gpu_selection_of_rows_that_a_sample_says_little_about(tokens, span):
    """Many equal scores at, above and below the threshold, at zero, among subnormals and at a mask; scores that
    change slowly along the row, in both directions of a missed floor; winners the sample has not seen."""
    import torch

    from ascendflow_b200 import neighbours

    rng = np.random.default_rng(span + tokens)
    scores = rng.normal(size=(tokens, span)).astype(np.float32)
    slow = np.convolve(rng.normal(size=tokens + span), np.exp(-np.arange(400) / 64), mode="same").astype(np.float32)
    place = np.arange(span)
    for token in range(tokens):
        few, kind = rng.choice(span, 400, replace=False), token % 14
        if kind == 0:
            scores[token] = np.maximum(scores[token] - 2.9, 0)              # fewer winners than TopK above zero
        elif kind == 1:
            scores[token] = np.maximum(scores[token] - 0.5, 0)
        elif kind == 2:
            scores[token] = 0.25
        elif kind == 3:
            scores[token] = np.where(np.isin(place, few), scores[token], -np.inf)
        elif kind == 4:
            scores[token] = np.round(scores[token] * 2) + np.float32(0.0)
        elif kind in (5, 6, 7):
            scores[token] = slow[token:token + span] + (0.01 * scores[token] if kind == 6 else 0)
        elif kind == 8:                                                      # the highest all in one place, away from a sample's start
            scores[token, 40:40 + 300] = 30 + rng.random(300)
        elif kind == 9:                                                      # far more high ones in the sampled head than elsewhere
            scores[token, :64] = 30
        elif kind == 10:                                                     # zeros of both signs and subnormals
            scores[token] = np.where(np.isin(place, few), np.float32(1e-41) * (place % 5), np.float32(-0.0))
        elif kind == 11:
            scores[token] = np.where(place % 3 == 0, np.float32(-1e-40), np.where(place % 3 == 1, np.float32(0.0), np.float32(-1.0)))
        elif kind == 12:                                                     # 400 above a plateau that is rare in the sample
            scores[token] = -np.abs(scores[token])
            scores[token, few] = 5
            scores[token, rng.choice(span, 120, replace=False)] = 4
        else:                                                                # ascending
            scores[token] = np.sort(scores[token])
    device = lambda array: torch.from_numpy(np.ascontiguousarray(array)).cuda()  # noqa: E731
    lengths = np.full(tokens, span, dtype=np.int32)
    lengths[::3] -= 5
    actual = neighbours.topk_indices(device(scores), device(np.arange(tokens + 1, dtype=np.int32)), device(lengths),
                                     device(np.zeros(tokens, dtype=np.int32)), ratio=1).cpu().numpy()[:, 0]
    bits = scores.view(np.uint32)
    for token in range(tokens):
        row = bits[token, :lengths[token]]
        key = np.where(row >> 31, ~row, row | 0x80000000)
        threshold = np.sort(key)[-512]
        above, equal = np.flatnonzero(key > threshold), np.flatnonzero(key == threshold)
        assert np.array_equal(actual[token], np.sort(np.concatenate([above, equal[:512 - len(above)]]))), (token, token % 14)
