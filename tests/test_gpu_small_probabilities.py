"""IEEE half keeps the precision of small probabilities: a row 2^-20 below the best one has a probability of
2^-12 (a normal number) while the reference stays eight binades below the best row, next to the sink, and of
2^-20 (four bits) where the reference moves up to that row although it need not."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SCALE_LOG2 = 512.0 ** -0.5 * 1.4426950408889634


@pytest.mark.parametrize("tokens", [1, 200])  # one cluster per token; persistent blocks
def test_probabilities_far_below_the_best_row_keep_their_bits(tokens):
    import torch

    from ascendflow_b200 import ops

    # Feature 0 makes the score, feature 1 is the output that is looked at: 0 in the best row, 1 in the
    # 511 others, whose score is about 20 (log2) lower.
    window, heads = 512, 64
    rows = np.zeros((window, 512), dtype=np.float16)
    rows[:, 0], rows[:, 1] = -0.9, 1.0
    rows[window - 125, :2] = 4.0, 0.0                    # in the first chunk: among the first 64 raw window rows
    q = np.zeros((tokens, heads, 512), dtype=np.float16)
    q[:, :, 0] = 63.0 + np.arange(heads) / 32.0
    best = q[0, :, 0].astype(np.float64) * 4.0 * SCALE_LOG2
    sinks = ((best - 7.75) / 1.4426950408889634).astype(np.float32)   # the reference: eight below the best

    i32 = lambda value: torch.tensor(np.ascontiguousarray(value), dtype=torch.int32, device="cuda")  # noqa: E731
    cache = torch.from_numpy(rows).cuda().view(window // 128, 128, 1, 512)
    indices = np.full((tokens, 1, 512), -1)
    indices[:, 0, :384] = np.arange(384)                 # the 384 rows in front of the window, uncompressed
    table = np.tile(np.arange(window // 128), (tokens, 1))
    out = torch.empty((tokens, heads, 512), dtype=torch.float16, device="cuda")
    ops.sparse_mla(torch.from_numpy(q).cuda(), cache, cache.clone(), i32(indices), i32(table), i32(table), i32(np.arange(tokens + 1)),
                   i32(np.full(tokens, window)), i32(np.full(tokens, window)), i32(np.zeros(tokens)), i32(np.zeros((tokens, 1))),
                   torch.from_numpy(sinks).cuda(), out)

    scores = q[0, :, 0].astype(np.float64)[:, None] * rows[:, 0].astype(np.float64)[None] * SCALE_LOG2
    weights = np.exp2(scores - best[:, None])
    expected = (weights * rows[:, 1]).sum(1) / (weights.sum(1) + np.exp2(sinks * 1.4426950408889634 - best))
    actual = out[:, :, 1].double().cpu().numpy()
    # P and the output are each rounded once to 11 bits: 2^-11 in all. The rest is FP32, where an
    # exponent of about 16 is off by 2^-20 at most. Four-bit probabilities are off by up to 2^-5.
    assert np.abs(actual / expected - 1).max() <= 2.0 ** -10
