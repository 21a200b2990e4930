"""The rounds in which the persistent blocks share a call's tokens: every token is worked on, once, whatever the
last round holds. A token's bits do not depend on its call, so a whole call must equal the same tokens in
pieces of one token per block (where five warps resolve every token; in the whole call one warp resolves most)."""

import numpy as np
import pytest

from oracle import sparse_mla_oracle as O
from tests import support as S
from tests.test_gpu_index_lists import KINDS, index_list

pytestmark = pytest.mark.gpu

PAGES = 1024  # of the pool that all requests share


def call(tokens):
    """One query per request, 1 to 2048 raw rows each."""
    import torch

    rng = np.random.default_rng(tokens)
    lengths = rng.integers(1, 2049, tokens).astype(np.int32)
    lengths[rng.integers(0, tokens, 8)] = 0  # and some that see nothing
    indices = np.full((tokens, 1, 512), -1, dtype=np.int32)
    for token, length in enumerate(lengths):
        take = min(512, int(length) // 2)
        if token % 3 == 0 and take:  # lists in no order, that end early, with entries behind the end or beyond the cutoff
            indices[token, 0] = index_list(rng, token // 3 % KINDS, int(length) // 2)
            continue
        indices[token, 0, :take] = np.sort(rng.choice(int(length) // 2, take, replace=False)) if take else []
    meta = {
        "cmp_sparse_indices": indices, "ori_block_table": rng.integers(0, PAGES, (tokens, 16)).astype(np.int32),
        "cmp_block_table": rng.integers(0, PAGES, (tokens, 16)).astype(np.int32),
        "cu_seqlens_q": np.arange(tokens + 1, dtype=np.int32), "seqused_ori_kv": lengths, "seqused_cmp_kv": lengths // 2,
        "cmp_residual_kv": lengths % 2, "ori_topk_length": np.zeros((tokens, 1), dtype=np.int32),
    }
    generator = torch.Generator(device="cuda")
    generator.manual_seed(tokens)
    normal = lambda *shape: torch.randn(shape, dtype=torch.bfloat16, device="cuda", generator=generator)  # noqa: E731
    tensors = {name: torch.from_numpy(np.ascontiguousarray(value)).cuda() for name, value in meta.items()}
    tensors.update(q=normal(tokens, 64, 512), ori_kv=normal(PAGES, 128, 1, 512), cmp_kv=normal(PAGES, 64, 1, 512),
                   sinks=torch.linspace(-3, 3, 64, device="cuda"))
    tensors["attention_out"] = torch.full_like(tensors["q"], float("nan"))
    return tensors, meta


def piece(tensors, first, count):
    """Tokens `first` ... as a call of their own, with an output of its own."""
    import torch

    part = {"attention_out": torch.full_like(tensors["attention_out"][first : first + count], float("nan"))}
    for name, value in tensors.items():
        if name == "attention_out":
            continue
        if name in ("ori_kv", "cmp_kv", "sinks"):
            part[name] = value
        elif name == "cu_seqlens_q":
            part[name] = value[: count + 1].contiguous()
        else:
            part[name] = value[first : first + count].contiguous()
    return part


@pytest.mark.parametrize("rounds,group,rest", [
    (4, 1, 1), (4, 1, -1),           # one token per block and round; one more, all but one more
    (4, 2, 0), (4, 2, 1), (4, 2, -1),  # groups of two: nothing left, dealt singly, in twos that do not go round
    (4, 3, 2), (5, 8, 1), (5, 8, -3),  # groups of three, and of eight (the largest): one each, seven or eight each
])
def test_every_token_of_every_round(rounds, group, rest):
    import torch

    from ascendflow_b200 import ops

    blocks = torch.cuda.get_device_properties(0).multi_processor_count
    tokens = rounds * group * blocks + (rest if rest >= 0 else group * blocks + rest)
    assert min(8, tokens // (4 * blocks)) == group
    tensors, meta = call(tokens)
    assert ops.kernel().bind(*(tensors[name] for name in S.TENSOR_ORDER))().status()[0] == 0
    assert not bool(tensors["attention_out"].isnan().any())
    policy = O.make_policy(tokens, tokens, ratio=2, max_seq=2048, dtype="bf16", blocks=PAGES)
    sample = [0, tokens // 2, tokens - 2, tokens - 1]
    actual = S.output_to_numpy(tensors["attention_out"], "bf16")
    S.assert_close(actual[sample], S.sampled_reference(tensors, meta, policy, sample), "rounds")
    for first in range(0, tokens, blocks):
        part = piece(tensors, first, min(blocks, tokens - first))
        ops.sparse_mla(*(part[name] for name in S.TENSOR_ORDER))
        whole = tensors["attention_out"][first : first + blocks]
        assert torch.equal(part["attention_out"].view(torch.int16), whole.view(torch.int16)), first
