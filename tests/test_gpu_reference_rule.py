"""The softmax's running reference moves when a chunk's best row is more than 15 binades above it, to 8 below that row, and
with a token's first chunk to a whole number of binades off that chunk's best row. Sinks from 70 binades above the best row to
40 below it, on both sides of every line; the best row alone, or behind an earlier one that the reference may have moved for.
And references that move chunk after chunk. All against 64 bits, in every feature."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SCALE_LOG2 = 512.0 ** -0.5 * 1.4426950408889634


@pytest.mark.parametrize("tokens", [1, 200])  # one cluster per token; persistent blocks
@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("gap", [0.0, 6.5, 9.0, 16.0, 23.0])
def test_sinks_far_below_the_best_row(tokens, dtype, gap):
    import torch

    from ascendflow_b200 import ops

    storage = getattr(torch, dtype)
    # Feature 0 makes the score, the others are the output that is looked at, each its own multiple of one value per row.
    # The early row is in the first chunk, `gap` binades below the best, which is among the last; the others weigh next to nothing.
    window, heads = 512, 64
    value = torch.ones(window)
    value[window - 125], value[350] = 0.75, 0.25
    rows = value[:, None] * (1 + torch.arange(512) % 31)[None] / 32
    rows[:, 0] = -3.0
    rows[window - 125, 0], rows[350, 0] = 4.0 * (1 - gap / 32.0), 4.0
    rows = rows.to(storage)
    assert torch.equal(rows[350, 1:].float() * 4, rows[0, 1:].float())  # (the products are exact)
    q = torch.zeros((tokens, heads, 512))
    q[:, :, 0] = 32.0 / (4.0 * SCALE_LOG2)
    q = q.to(storage)
    best = q[0, :, 0].double() * 4.0 * SCALE_LOG2
    below = torch.cat([torch.linspace(-70.0, -1.5, 16), torch.linspace(-1.0, 40.0, heads - 16)])
    sinks = ((best - below) / 1.4426950408889634).float()

    i32 = lambda value: torch.tensor(np.ascontiguousarray(value), dtype=torch.int32, device="cuda")  # noqa: E731
    cache = rows.cuda().view(window // 128, 128, 1, 512)
    indices = np.full((tokens, 1, 512), -1)
    indices[:, 0, :384] = np.arange(384)                 # the 384 rows in front of the window, uncompressed
    table = np.tile(np.arange(window // 128), (tokens, 1))
    out = torch.empty((tokens, heads, 512), dtype=storage, device="cuda")
    ops.sparse_mla(q.cuda(), cache, cache.clone(), i32(indices), i32(table), i32(table), i32(np.arange(tokens + 1)),
                   i32(np.full(tokens, window)), i32(np.full(tokens, window)), i32(np.zeros(tokens)), i32(np.zeros((tokens, 1))),
                   sinks.cuda(), out)

    scores = q[0, :, 0].double()[:, None] * rows[:, 0].double()[None] * SCALE_LOG2
    weights = torch.exp2(scores - best[:, None])
    expected = weights @ rows[:, 1:].double() / (weights.sum(1) + torch.exp2(sinks.double() * 1.4426950408889634 - best))[:, None]
    actual = out[:, :, 1:].double().cpu()
    # P and the output are each rounded once, to 11 or 8 bits: an ulp in all. The rest is FP32 (exponents of up to 40:
    # 2^-18). A half that overflowed would be infinite, a reference that was not followed a power of two off. Below a sink far
    # above the rows a half's steps are of 2^-24: half a step for the output and for either of two probabilities.
    assert ((actual - expected).abs() <= expected * 2.0 ** (-10 if dtype == "float16" else -7) + 1.5 * 2.0**-24).all()


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("tokens", [1, 33, 320])  # one cluster per token; persistent blocks of up to three
def test_references_that_move_at_many_chunks(tokens, dtype):
    import torch

    from ascendflow_b200 import ops

    storage = getattr(torch, dtype)
    generator = torch.Generator().manual_seed(tokens)
    normal = lambda *shape: torch.randn(shape, generator=generator)  # noqa: E731
    # Scores rise by up to twelve binades from chunk to chunk through the window's two and the list's eight, and where the list
    # begins at another row of the cache for another token, fall once in between. Heads differ by how much.
    heads, raw, listed = 64, 128, 512
    rows = normal(listed + raw, 512)
    rows[:, 0] = torch.cat([torch.arange(listed) // 64 + 2, torch.arange(raw) // 64]) / 4.0 + 0.01 * normal(listed + raw)
    rows = rows.to(storage)
    q = 0.05 * normal(tokens, heads, 512)
    q[:, :, 0] = (2 + 10 * torch.rand((tokens, heads), generator=generator)) * 4.0 / SCALE_LOG2
    q = q.to(storage)
    sinks = -20.0 + 10.0 * normal(heads)
    first = torch.randint(0, 8, (tokens,), generator=generator) * (torch.arange(tokens) % 2) * 64
    indices = (torch.arange(listed)[None] + first[:, None]) % listed

    def call(count):
        i32 = lambda given: given.to(torch.int32).cuda()  # noqa: E731
        pages = (listed + raw) // 128
        table = i32(torch.arange(pages).expand(count, pages).contiguous())
        length = torch.full((count,), listed + raw)
        cache = rows.cuda().view(pages, 128, 1, 512)
        out = torch.full((count, heads, 512), float("nan"), dtype=storage, device="cuda")
        ops.sparse_mla(q[:count].cuda(), cache, cache.clone(), i32(indices[:count, None]), table, table.clone(), i32(torch.arange(count + 1)),
                       i32(length), i32(length), i32(0 * length), i32(torch.zeros(count, 1)), sinks.cuda(), out)
        return out.cpu()

    actual = call(tokens)
    if tokens > 33:  # the same tokens in the other kernel
        assert torch.equal(call(20).view(torch.int16), actual[:20].view(torch.int16))
    x = rows.double()
    scores = (q.double() @ x.T) * SCALE_LOG2
    sink = (sinks.double() * 1.4426950408889634)[None, :, None]
    best = scores.amax(2, keepdim=True)
    weights = torch.exp2(scores - best)
    total = weights.sum(2, keepdim=True) + torch.exp2(sink - best)
    expected, size = weights @ x / total, weights @ x.abs() / total

    order = torch.cat([torch.arange(raw).expand(tokens, raw) + listed, indices], 1)  # the order of the slots
    chunks = torch.gather(scores, 2, order[:, None].expand_as(scores)).view(tokens, heads, 10, 64).amax(3)
    reference, moves = sink[..., 0].expand(tokens, heads), 0
    for chunk in range(10):
        moved = chunks[..., chunk] > reference + 15
        moves = moves + (moved & (chunk > 0))
        reference = torch.where(moved, chunks[..., chunk] - 8, reference)
    assert (moves >= 3).double().mean() > 0.5 and int(moves.max()) >= 6

    # P and the output are each rounded once to 11 or 8 bits. Scores of a hundred binades in FP32 are off by 2^-17 of themselves at most
    # (512 products), a weight then by 2^-11 with the reference's as much. Half has steps of 2^-24 for what lies below the best row
    # (or a sink above it).
    unit = 2.0 ** (-11 if dtype == "float16" else -8)
    tolerance = unit * (expected.abs() + size) + 2.0**-10 * size + (2.0**-25 * x.abs().sum(0) if dtype == "float16" else 0)
    assert ((actual.double() - expected).abs() <= tolerance).all()


@pytest.mark.parametrize("dtype,scale", [("bfloat16", 1.0), ("bfloat16", 3.0), ("float16", 1.0), ("float16", 3.0)])
@pytest.mark.parametrize("tokens", [16, 320])
def test_the_error_is_that_of_two_roundings(tokens, dtype, scale):
    """Against 64 bits, by the 2-norm: P and the output are rounded once each, and nothing else shows."""
    import torch

    from ascendflow_b200 import ops

    storage = getattr(torch, dtype)
    generator = torch.Generator().manual_seed(tokens)
    normal = lambda *shape: torch.randn(shape, generator=generator)  # noqa: E731
    rows, q, sinks = normal(4096, 512).to(storage), (scale * normal(tokens, 64, 512)).to(storage), normal(64)
    indices = torch.stack([torch.randperm(4096 - 128, generator=generator)[:512].sort().values for _ in range(tokens)])
    i32 = lambda given: given.to(torch.int32).cuda()  # noqa: E731
    table, length = i32(torch.arange(32).expand(tokens, 32).contiguous()), torch.full((tokens,), 4096)
    cache = rows.cuda().view(32, 128, 1, 512)
    out = torch.empty((tokens, 64, 512), dtype=storage, device="cuda")
    ops.sparse_mla(q.cuda(), cache, cache.clone(), i32(indices[:, None]), table, table.clone(), i32(torch.arange(tokens + 1)), i32(length),
                   i32(length), i32(0 * length), i32(torch.zeros(tokens, 1)), sinks.cuda(), out)
    expected = torch.empty((tokens, 64, 512), dtype=torch.float64)
    for token in range(tokens):
        x = torch.cat([rows[-128:], rows[indices[token]]]).double()
        scores = q[token].double() @ x.T * 512.0**-0.5
        weights = torch.cat([scores, sinks.double()[:, None]], 1).softmax(1)[:, :-1]
        expected[token] = weights @ x
    error = float((out.double().cpu() - expected).norm() / expected.norm())
    # A value whose logarithm is spread evenly is off by 2^-7 / sqrt(12) (bf16) or 2^-10 / sqrt(12) (half) of its binade's
    # lower end, by 0.7355 of that relative to itself; two of them, independent.
    one = 2.0 ** (-10 if dtype == "float16" else -7) / 12**0.5 * 0.7355
    assert error <= 2**0.5 * one, (error, 2**0.5 * one)
