"""The softmax's running reference moves when a chunk's best row is more than 15 binades above it, to 8 below that row, and
with a token's first chunk to a whole number of binades off that chunk's best row. Sinks from 70 binades above the best row to
40 below it, on both sides of every line; the best row alone, or behind an earlier one that the reference may have moved for."""

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
    # Feature 0 makes the score, feature 1 is the output that is looked at. The early row is in the first chunk,
    # `gap` binades below the best, which is among the last; the others weigh next to nothing.
    window, heads = 512, 64
    rows = torch.zeros((window, 512))
    rows[:, 0], rows[:, 1] = -3.0, 1.0
    rows[window - 125, :2] = torch.tensor([4.0 * (1 - gap / 32.0), 0.75])
    rows[350, :2] = torch.tensor([4.0, 0.25])
    rows = rows.to(storage)
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
    expected = (weights * rows[:, 1].double()).sum(1) / (weights.sum(1) + torch.exp2(sinks.double() * 1.4426950408889634 - best))
    actual = out[:, :, 1].double().cpu()
    # P and the output are each rounded once, to 11 or 8 bits: an ulp in all. The rest is FP32 (exponents of up to 40:
    # 2^-18). A half that overflowed would be infinite, a reference that was not followed a power of two off. Below a sink far
    # above the rows a half's steps are of 2^-24: half a step for the output and for either of two probabilities.
    assert ((actual - expected).abs() <= expected * 2.0 ** (-10 if dtype == "float16" else -7) + 1.5 * 2.0**-24).all()
