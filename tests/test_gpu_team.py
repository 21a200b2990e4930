"""The cluster kernel for calls of few tokens: the same bits as the persistent kernel for every number of
chunks, with and without a reference that moves late, and against the FP32 reference.

A call of few tokens and the same tokens at the head of a call too large for the cluster kernel must
agree bit for bit."""

import numpy as np
import pytest

from oracle import sparse_mla_oracle as O
from tests import support as S

pytestmark = pytest.mark.gpu

MANY = 160  # more tokens than any device has room for clusters


def call(rng, lengths, ratio, dtype, scale):
    """One query per request, `lengths` raw rows each; q scaled so that references move late."""
    policy = O.make_policy(len(lengths), len(lengths), ratio=ratio, max_seq=2048, dtype=dtype)
    import torch

    lengths = np.asarray(lengths, dtype=np.int32)
    tokens = len(lengths)
    indices = np.full((tokens, 1, 512), -1, dtype=np.int32)
    for token, length in enumerate(lengths):
        take = min(512, int(length) // ratio)
        indices[token, 0, :take] = np.sort(rng.choice(int(length) // ratio, take, replace=False)) if take else []
    table = rng.permutation(tokens * 16).reshape(tokens, 16).astype(np.int32)
    meta = {
        "cmp_sparse_indices": indices, "ori_block_table": table, "cmp_block_table": table[:, ::-1].copy(),
        "cu_seqlens_q": np.arange(tokens + 1, dtype=np.int32), "seqused_ori_kv": lengths, "seqused_cmp_kv": lengths // ratio,
        "cmp_residual_kv": lengths % ratio, "ori_topk_length": np.zeros((tokens, 1), dtype=np.int32),
    }
    generator = torch.Generator(device="cuda")
    generator.manual_seed(int(rng.integers(1 << 30)))
    storage = S.torch_dtype(dtype)
    normal = lambda *shape: torch.randn(shape, device="cuda", generator=generator).to(storage)  # noqa: E731
    tensors = {name: torch.from_numpy(np.ascontiguousarray(value)).cuda() for name, value in meta.items()}
    tensors.update(q=normal(tokens, 64, 512) * scale, ori_kv=normal(tokens * 16, 128, 1, 512),
                   cmp_kv=normal(tokens * 16, 128 // ratio, 1, 512), sinks=torch.linspace(-3, 3, 64, device="cuda"))
    tensors["attention_out"] = torch.full_like(tensors["q"], float("nan"))
    return tensors, meta, policy


def head(tensors, tokens):
    """The first `tokens` one-query requests as a call of their own (same caches)."""
    part = {}
    for name, value in tensors.items():
        part[name] = value if name in ("ori_kv", "cmp_kv", "sinks") else value[: tokens + (name == "cu_seqlens_q")].contiguous()
    part["attention_out"] = part["attention_out"].clone()
    return part


@pytest.mark.parametrize("ratio,dtype,scale", [(2, "bf16", 1.0), (2, "bf16", 6.0), (1, "f16", 1.0), (1, "f16", 6.0)])
def test_few_tokens_give_the_bits_of_many(ratio, dtype, scale):
    import torch

    from ascendflow_b200 import ops

    rng = np.random.default_rng(int(scale) * 10 + ratio)
    # every number of live chunks from none to ten, ragged tails
    lengths = [1, 0, 63, 64, 65, 128, 129, 200, 255, 256, 300, 384, 500, 640, 800, 1024, 1100, 1500, 2048] * 9
    tensors, _, _ = call(rng, lengths[:MANY], ratio, dtype, scale)
    ops.sparse_mla(*(tensors[name] for name in S.TENSOR_ORDER))
    for tokens in (1, 2, 3, 16, 18, 32, 33, 34, 40):
        part = head(tensors, tokens)
        ops.sparse_mla(*(part[name] for name in S.TENSOR_ORDER))
        torch.cuda.synchronize()
        assert torch.equal(part["attention_out"].view(torch.int16), tensors["attention_out"][:tokens].view(torch.int16)), tokens


def test_a_token_without_visible_rows_and_the_fp32_reference():
    import torch

    from ascendflow_b200 import ops

    rng = np.random.default_rng(3)
    tensors, meta, policy = call(rng, [1500, 0, 700, 90, 2048], 2, "bf16", 1.0)
    binding = ops.kernel().bind(*(tensors[name] for name in S.TENSOR_ORDER))()
    assert binding.status()[0] == 0
    actual = S.output_to_numpy(tensors["attention_out"], "bf16")
    S.assert_close(actual, S.sampled_reference(tensors, meta, policy, list(range(5))), "team")
    assert not actual[1].any()


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
def test_an_output_that_starts_between_sectors(dtype):
    """Whole sectors are stored where the output starts on one, halves of them otherwise: the same bits, and nothing beside them."""
    import torch

    from ascendflow_b200 import ops

    tensors, _, _ = call(np.random.default_rng(5), [1500, 90, 0, 640], 2, dtype, 1.0)
    ops.sparse_mla(*(tensors[name] for name in S.TENSOR_ORDER))
    count = tensors["attention_out"].numel()
    for offset in (8, 16, 24):  # elements of two bytes
        room = torch.full((count + 48,), 7.0, dtype=tensors["attention_out"].dtype, device="cuda")
        start = offset + (-room.data_ptr() // 2) % 16
        moved = dict(tensors, attention_out=room[start : start + count].view(tensors["attention_out"].shape))
        assert moved["attention_out"].data_ptr() % 32 == offset * 2 % 32
        ops.sparse_mla(*(moved[name] for name in S.TENSOR_ORDER))
        torch.cuda.synchronize()
        assert torch.equal(moved["attention_out"].view(torch.int16), tensors["attention_out"].view(torch.int16)), offset
        assert (room[:start] == 7).all() and (room[start + count :] == 7).all(), offset
