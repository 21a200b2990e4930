"""The native host side against the Python front end: same results for what it accepts, the front end's
errors for what it does not, on streams and threads."""

import numpy as np
import pytest

from oracle import sparse_mla_oracle as O
from tests import support as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def call():
    policy = O.make_policy(4, 16, max_seq=4096, blocks=128)
    return S.to_device(O.validation_inputs(policy, "mixed"), policy)[0]


def arguments(tensors, **changed):
    return [changed.get(name, tensors[name]) for name in S.TENSOR_ORDER]


@pytest.mark.parametrize("entry", ["function", "op"])
@pytest.mark.parametrize("name,change,message", [
    ("q", lambda t: t.float(), "dtype differs"),
    ("sinks", lambda t: t[:32], "shape differs"),
    ("cmp_kv", lambda t: t[:, :32].contiguous(), "contract differs"),
    ("cu_seqlens_q", lambda t: t.cpu(), "CUDA tensor"),
    ("ori_topk_length", lambda t: t.view(-1), "rank differs"),
    ("attention_out", None, "disjoint"),
    ("cmp_sparse_indices", lambda t: t.repeat(1, 1, 2)[:, :, ::2], "contiguous"),
])
def test_refused_arguments_raise_the_front_ends_error(call, entry, name, change, message):
    import torch

    from ascendflow_b200 import ops
    from ascendflow_b200.diagnostics import CompileError

    ops.sparse_mla(*arguments(call))  # the entry points are connected
    wrong = arguments(call, **{name: call["q"] if change is None else change(call[name])})
    with pytest.raises(CompileError, match=message):
        (ops.sparse_mla if entry == "function" else torch.ops.ascendflow_b200.sparse_mla)(*wrong)


def test_streams_and_threads_get_the_same_output(call):
    import threading

    import torch

    from ascendflow_b200 import ops

    binding = ops.kernel().bind(*arguments(call))
    binding()
    torch.cuda.synchronize()
    expected = call["attention_out"].clone()
    outputs = {}

    def work(key):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            mine = torch.empty_like(call["attention_out"])
            for _ in range(20):
                torch.ops.ascendflow_b200.sparse_mla(*arguments(call, attention_out=mine))
        stream.synchronize()
        outputs[key] = mine

    threads = [threading.Thread(target=work, args=(key,)) for key in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert all(torch.equal(outputs[key], expected) for key in range(4))


def test_op_counts_as_a_mutation_and_has_no_gradient(call):
    import torch

    out = torch.empty_like(call["attention_out"])
    version = out._version
    torch.ops.ascendflow_b200.sparse_mla(*arguments(call, attention_out=out))
    assert out._version == version + 1
    q = call["q"].clone().requires_grad_()
    torch.ops.ascendflow_b200.sparse_mla(*arguments(call, q=q, attention_out=out))
    with pytest.raises(RuntimeError):
        out.sum().backward()


def test_append_reports_a_bad_page_once_and_is_clean_afterwards():
    import torch

    from ascendflow_b200 import neighbours

    cache = torch.zeros((4, 128, 1, 512), dtype=torch.bfloat16, device="cuda")
    rows = torch.ones((3, 512), dtype=torch.bfloat16, device="cuda")
    cu = torch.tensor([0, 3], dtype=torch.int32, device="cuda")
    table = torch.tensor([[0, 1, 2, 3]], dtype=torch.int32, device="cuda")
    for length, code in ((3, 0), (514, 1), (512, 0)):
        status = neighbours.cache_append(rows, cache, table, cu, torch.tensor([length], dtype=torch.int32, device="cuda"))
        assert status[0] == code and len(status) == 8
        if code:
            assert status[1:3] in ((1, 512), (2, 513))
    assert np.array_equal(cache.view(512, 512)[:, 0].float().cpu().numpy().nonzero()[0], [0, 1, 2, 509, 510, 511])


def test_append_reports_on_side_streams_neither_stay_nor_vanish():
    """Bad and good appends in turn on streams that do not wait for the default stream, while that one is
    busy: each call's report is its own. Blocks are new on every other round."""
    import torch

    from ascendflow_b200 import host, neighbours

    cache = torch.zeros((4, 128, 1, 512), dtype=torch.bfloat16, device="cuda")
    rows = torch.ones((3, 512), dtype=torch.bfloat16, device="cuda")
    cu = torch.tensor([0, 3], dtype=torch.int32, device="cuda")
    table = torch.tensor([[0, 1, 2, 3]], dtype=torch.int32, device="cuda")
    lengths = {code: torch.tensor([length], dtype=torch.int32, device="cuda") for code, length in ((0, 100), (1, 515))}
    streams = [torch.cuda.Stream() for _ in range(3)]
    work = torch.zeros(1 << 24, device="cuda")
    torch.cuda.synchronize()
    for turn in range(30):
        if turn % 2 == 0:
            host.calls.release_workspaces()
        for _ in range(4):
            work.add_(1)
        with torch.cuda.stream(streams[turn % 3]):
            code = (turn % 5) % 2
            status = neighbours.cache_append(rows, cache, table, cu, lengths[code])
            assert status[0] == code
            assert status[1:3] in ((0, 512), (1, 513), (2, 514)) if code else status == (0,) * 8


def with_a_bad_page(call):
    """The call with page numbers in the first request's table that no cache has, and as it was."""
    table = call["ori_block_table"].clone()
    table[0, :] = 1 << 20
    return arguments(call, ori_block_table=table), arguments(call)


@pytest.mark.parametrize("entry", ["function", "op"])
def test_status_reports_a_bad_page_once(call, entry):
    import torch

    from ascendflow_b200 import ops

    launch = ops.sparse_mla if entry == "function" else torch.ops.ascendflow_b200.sparse_mla
    bad, good = with_a_bad_page(call)
    ops.status()                            # what other tests' calls on this stream have left
    side = torch.cuda.Stream()
    for stream in (torch.cuda.current_stream(), side):
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            for arguments_, code in ((good, 0), (bad, 1), (good, 0), (bad, 1), (bad, 1)):
                launch(*arguments_)
                status = ops.status()
                assert status[0] == code and len(status) == 8
                assert ops.status() == (0,) * 8
                assert code or status == (0,) * 8
            launch(*bad)
            launch(*good)
            assert ops.status()[0] == 1     # a good call does not take a report away
    torch.cuda.synchronize()


def test_captured_calls_report_and_outlive_kept_blocks(call):
    """A first call on a capturing stream, replayed after every kept block has been given back and its memory reused."""
    import torch

    from ascendflow_b200 import host, ops

    bad, good = with_a_bad_page(call)
    ops.sparse_mla(*good)
    expected = call["attention_out"].clone()
    ops.status()
    graphs = []
    for arguments_ in (good, bad):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            ops.sparse_mla(*arguments_)
        graphs.append(graph)
    host.calls.release_workspaces()
    filled = [torch.full((1024,), 0x5A, dtype=torch.uint8, device="cuda") for _ in range(64)]
    for graph, code in zip((graphs[0], graphs[1], graphs[0], graphs[1]), (0, 1, 0, 1)):
        call["attention_out"].zero_()
        graph.replay()
        status = ops.status()
        assert status[0] == code and (code or torch.equal(call["attention_out"], expected))
    ops.sparse_mla(*good)
    assert ops.status() == (0,) * 8
    assert all(bool((block == 0x5A).all()) for block in filled)
