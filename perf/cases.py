"""The calls this library is measured on, as a serving program makes them.

Four kinds of call, each through a public entry point:

  attention  one sparse MLA call (`ops.sparse_mla`, the registered torch op, or the upstream-shaped
             `upstream.sparse_flash_mla`, which also allocates the output)
  select     index scores -> `cmp_sparse_indices` (`neighbours.topk_indices`)
  append     a step's new rows -> the paged cache (`neighbours.cache_append`)
  layer      what one layer does in a serving step: append, select, attention

A case gives sizes and options only. Request lengths follow from the case (so the work of a pass
does), everything else (cache contents, page permutations, indices, scores) from the seed.
"""

import math
import random

import torch

from ascendflow_b200 import neighbours, ops, upstream

HEADS, FEATURES, WINDOW, TOPK, PAGE = 64, 512, 128, 512, 128
ROW = FEATURES * 2
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16}


def _case(kind, requests, queries, context, **options):
    # ragged: requests of different chunk and context lengths (`queries` and `context` are the
    #         longest), as continuous batching makes them; otherwise all requests are alike
    # narrow: per-token window lengths below 128 (`ori_topk_length`)
    # coarse: index scores that carry 8 mantissa bits (a 16-bit index network): many exact ties
    case = {"kind": kind, "requests": requests, "queries": queries, "context": context, "ratio": 2,
            "dtype": "bf16", "entry": "function", "ragged": False, "narrow": False, "coarse": False}
    case.update(options)
    return case


def listed():
    return [
        # One user, one token: what an interactive session waits for between two tokens.
        _case("attention", 1, 1, 8192, name="decode_1x1_8k"),
        # A small batch with one speculated token each, called through the registered op.
        _case("attention", 8, 2, 16384, entry="op", name="decode_8x2_16k"),
        # Draft verification (five drafts and one token) for 64 and 128 requests at 128K: the two
        # decode rows of the benchmark.
        _case("attention", 64, 6, 131072, name="decode_64x6_128k"),
        _case("attention", 128, 6, 131072, name="decode_128x6_128k"),
        # A short chunk at the end of a 4K context: the benchmark's CPU-reference shape.
        _case("attention", 1, 256, 4096, name="prefill_256_4k"),
        # The benchmark's two prefill rows: the last 8K of a 32K context, and all of a 32K prompt.
        _case("attention", 1, 8192, 32768, name="prefill_8k_32k"),
        _case("attention", 1, 32768, 32768, name="prefill_32k_32k"),
        # Continuous batching: prompt chunks and decode tokens of odd lengths in one call, IEEE half,
        # uncompressed cache (ratio 1), narrowed windows, through the upstream-shaped adapter.
        _case("attention", 23, 700, 20011, ratio=1, dtype="f16", entry="upstream", ragged=True, narrow=True,
              name="mixed_23_f16_c1"),
        # Index selection for the large decode batch and for a prefill chunk.
        _case("select", 128, 6, 131072, name="select_128x6_128k"),
        _case("select", 1, 8192, 32768, coarse=True, name="select_8k_32k"),
        # A prefill chunk's new rows into the cache.
        _case("append", 1, 8192, 32768, name="append_8k"),
        # One layer of an ordinary decode step: 16 requests of different ages, one token each.
        _case("layer", 16, 1, 32768, ragged=True, name="layer_16x1_32k"),
    ]


def _log(rng, low, high):
    """A whole number, spread evenly over the logarithm."""
    return min(high, max(low, int(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng):
    kind = rng.choice(["attention"] * 6 + ["select"] * 2 + ["append"] + ["layer"] * 2)
    ratio = rng.choice([2, 2, 2, 1])
    dtype = rng.choice(["bf16", "bf16", "f16"])
    ragged = rng.random() < 0.4
    if kind == "attention" and rng.random() < 0.5 or kind == "select" and rng.random() < 0.5:  # prefill
        requests, queries = _log(rng, 1, 24), _log(rng, 32, 16384)
        queries = min(queries, 24576 // requests)
        context = _log(rng, max(queries, 1024), 65536)
    elif kind == "append":
        requests, queries = _log(rng, 1, 64), _log(rng, 1, 8192)
        queries = min(queries, 32768 // requests)
        context = _log(rng, max(queries, 256), max(queries, 524288 // requests))
    else:  # decode
        requests, queries = _log(rng, 1, 128), rng.randint(1, 6)
        context = _log(rng, 1024, 131072)
    if kind == "layer":
        context = min(context, 1048576 // requests)
    if kind == "select":  # at most 2 GiB of scores
        context = min(context, (1 << 29) // (requests * queries) * ratio)
        queries = min(queries, context)
    # at most the caches of the largest decode case
    context = max(queries, min(context, 128 * 131072 * 3 // (2 * requests * (1 + ratio % 2))))
    return _case(kind, requests, queries, context, ratio=ratio, dtype=dtype, ragged=ragged,
                 entry=rng.choice(["function", "function", "op", "upstream"]) if kind == "attention" else "function",
                 narrow=kind == "attention" and rng.random() < 0.2,
                 coarse=kind in ("select", "layer") and rng.random() < 0.5)


def _lengths(case):
    """Query tokens and context of every request. The first is the longest; in a ragged call about
    half of the others decode one token and the rest bring chunks."""
    counts, lengths = [case["queries"]], [case["context"]]
    rng = random.Random("%d %d %d" % (case["requests"], case["queries"], case["context"]))
    for _ in range(case["requests"] - 1):
        if case["ragged"]:
            counts.append(1 if rng.random() < 0.5 else _log(rng, 1, case["queries"]))
            lengths.append(_log(rng, min(max(counts[-1], 64), case["context"]), case["context"]))
        else:
            counts.append(case["queries"])
            lengths.append(case["context"])
    return counts, lengths


def _narrowed(token):
    return (token * 37 + 11) % 160  # 0: all 128 rows; above 128: no narrowing either


def _generator(seed):
    generator = torch.Generator(device="cuda")
    generator.manual_seed(seed)
    return generator


def _normal(shape, dtype, generator):
    return torch.randn(shape, dtype=dtype, device="cuda", generator=generator)


def _per_token(case):
    """cu_seqlens_q and, per token, its request and right edge (rows of the raw cache it sees)."""
    counts, lengths = _lengths(case)
    count = torch.tensor(counts, device="cuda")
    cu = torch.cat([torch.zeros(1, dtype=torch.long, device="cuda"), count.cumsum(0)])
    request = torch.repeat_interleave(torch.arange(len(counts), device="cuda"), count)
    offset = torch.arange(len(request), device="cuda") - cu[request]
    right = torch.tensor(lengths, device="cuda")[request] - count[request] + offset + 1
    return cu.to(torch.int32), request, right


def _indices(case, right, generator):
    """For every token, 512 distinct uniform draws from its visible compressed rows (all of them
    where there are fewer), ascending, -1 padded."""
    cutoff = right // case["ratio"]
    out = torch.full((len(right), 1, TOPK), -1, dtype=torch.int32, device="cuda")
    span = max(int(cutoff.max()), 1)
    step = max(1, (1 << 27) // span)
    for first in range(0, len(right), step):
        edge = cutoff[first : first + step, None]
        keys = torch.rand((len(edge), span), device="cuda", generator=generator)
        keys.masked_fill_(torch.arange(span, device="cuda") >= edge, 2.0)
        take = min(TOPK, span)
        picked = keys.topk(take, dim=1, largest=False, sorted=False).indices
        picked = torch.where(picked < edge, picked, 1 << 30).sort(dim=1).values
        out[first : first + step, 0, :take] = torch.where(picked < (1 << 30), picked, -1).to(torch.int32)
    return out


def _tables(case, generator):
    """Page numbers of every request: pages are handed out from one pool in random order."""
    pages = -(-case["context"] // PAGE)
    blocks = case["requests"] * pages
    return torch.randperm(blocks, device="cuda", generator=generator).to(torch.int32).view(case["requests"], pages), blocks


def _scores(case, tokens, generator):
    span = -(-(case["context"] // case["ratio"]) // 4) * 4
    scores = _normal((tokens, max(span, 4)), torch.float32, generator)
    return scores.to(torch.bfloat16).to(torch.float32) if case["coarse"] else scores


def prepare(case, seed):
    generator = _generator(seed)
    counts, lengths = _lengths(case)
    dtype, ratio, kind = DTYPES[case["dtype"]], case["ratio"], case["kind"]
    cu, request, right = _per_token(case)
    tokens = len(request)
    length = torch.tensor(lengths, dtype=torch.int32, device="cuda")
    state = {"case": case, "cu_seqlens_q": cu, "seqused_ori_kv": length, "seqused_cmp_kv": length // ratio,
             "cmp_residual_kv": length % ratio}
    if kind in ("select", "layer"):
        state["scores"] = _scores(case, tokens, generator)
    if kind == "select":
        return state
    state["ori_block_table"], blocks = _tables(case, generator)
    state["ori_kv"] = _normal((blocks, PAGE, 1, FEATURES), dtype, generator)
    if kind in ("append", "layer"):
        state["new_rows"] = _normal((tokens, FEATURES), dtype, generator)
    if kind == "append":
        return state
    state["cmp_block_table"], blocks = _tables(case, generator)
    state["cmp_kv"] = _normal((blocks, PAGE // ratio, 1, FEATURES), dtype, generator)
    state["q"] = _normal((tokens, HEADS, FEATURES), dtype, generator)
    if kind == "attention":
        state["cmp_sparse_indices"] = _indices(case, right, generator)
    narrow = _narrowed(torch.arange(tokens, device="cuda")) if case["narrow"] else torch.zeros(tokens, device="cuda")
    state["ori_topk_length"] = narrow.to(torch.int32).view(tokens, 1).contiguous()
    state["sinks"] = _normal((HEADS,), torch.float32, generator)
    if case["entry"] != "upstream":
        state["attention_out"] = torch.empty_like(state["q"])
    return state


def _attention(state, indices):
    arguments = (state["q"], state["ori_kv"], state["cmp_kv"], indices, state["ori_block_table"], state["cmp_block_table"],
                 state["cu_seqlens_q"], state["seqused_ori_kv"], state["seqused_cmp_kv"], state["cmp_residual_kv"],
                 state["ori_topk_length"], state["sinks"])
    entry = state["case"]["entry"]
    if entry == "upstream":
        return upstream.sparse_flash_mla(*arguments)
    if entry == "op":
        torch.ops.ascendflow_b200.sparse_mla(*arguments, state["attention_out"])
        return state["attention_out"]
    return ops.sparse_mla(*arguments, state["attention_out"])


def _select(state):
    return neighbours.topk_indices(state["scores"], state["cu_seqlens_q"], state["seqused_cmp_kv"],
                                   state["cmp_residual_kv"], ratio=state["case"]["ratio"])


def _append(state):
    return neighbours.cache_append(state["new_rows"], state["ori_kv"], state["ori_block_table"], state["cu_seqlens_q"],
                                   state["seqused_ori_kv"])


def run(state):
    kind = state["case"]["kind"]
    if kind == "attention":
        return _attention(state, state["cmp_sparse_indices"])
    if kind == "select":
        return _select(state)
    if kind == "append":
        return {"status": _append(state), "cache": state["ori_kv"]}
    status = _append(state)
    indices = _select(state)
    return {"status": status, "cache": state["ori_kv"], "indices": indices, "out": _attention(state, indices)}


def work(case):
    counts, lengths = _lengths(case)
    tokens, ratio, kind = sum(counts), case["ratio"], case["kind"]
    live = distinct = visible_scores = token = 0
    for count, length in zip(counts, lengths):
        for j in range(count):
            right = length - count + j + 1
            narrow = _narrowed(token) if case["narrow"] else 0
            live += min(right, WINDOW, narrow if narrow > 0 else WINDOW) + min(TOPK, right // ratio)
            visible_scores += right // ratio
            token += 1
        # rows that at least one of a request's tokens reads: the union of the windows, and the
        # expected union of `count` draws of 512 out of the visible compressed rows
        visible = length // ratio
        missed = (1 - min(1.0, TOPK / visible)) ** count if visible else 0.0
        distinct += min(length, count - 1 + WINDOW) + round(visible * (1 - missed))
    small = 4 * (len(counts) * 4 + tokens) + 8 * sum(-(-length // PAGE) for length in lengths)
    attention = {"bytes": distinct * ROW + 2 * tokens * HEADS * ROW + tokens * TOPK * 4 + small,
                 "flops": 4 * HEADS * FEATURES * live}
    select = {"bytes": 4 * visible_scores + tokens * TOPK * 4 + 16 * len(counts), "flops": 0}
    append = {"bytes": 2 * tokens * ROW + 4 * (tokens + 2 * len(counts)), "flops": 0}
    parts = {"attention": [attention], "select": [select], "append": [append], "layer": [append, select, attention]}[kind]
    return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}


def tolerance(case):
    # Selection and append move whole values. Attention rounds its probabilities and its output to
    # the storage type (half an ulp: 2^-9 for bf16, 2^-12 for half) and sums in FP32; `max` allows
    # an output ulp on top of five standard deviations of the probabilities' rounding.
    if case["kind"] in ("select", "append"):
        return "exact"
    if case["dtype"] == "bf16":
        return {"rel": 5e-3, "max": 4e-2, "differ": 0.0}
    return {"rel": 1e-3, "max": 8e-3, "differ": 0.0}
