"""The native host side where there is no device: what the registered op does with tensors of other backends and
under torch's transforms, and whose errors the functions raise."""

import pytest
import torch

from ascendflow_b200 import host, neighbours, ops
from ascendflow_b200.diagnostics import CompileError


def arguments(device):
    shapes = [(4, 64, 512), (8, 128, 1, 512), (8, 64, 1, 512), (4, 1, 512), (2, 3), (2, 3), (3,), (2,), (2,), (2,), (4, 1), (64,), (4, 64, 512)]
    types = [torch.bfloat16] * 3 + [torch.int32] * 8 + [torch.float32, torch.bfloat16]
    return [torch.empty(shape, dtype=dtype, device=device) for shape, dtype in zip(shapes, types)]


op = torch.ops.ascendflow_b200.sparse_mla


@pytest.mark.parametrize("tracked", [0, 12])  # q; the output
def test_op_cannot_be_differentiated_by_functorch(tracked):
    def loss(factor):
        call = arguments("meta")
        call[tracked] = call[tracked] * factor
        op(*call)
        return call[12].sum()

    with pytest.raises(RuntimeError):
        torch.func.grad(loss)(torch.ones((), dtype=torch.bfloat16, device="meta"))


def test_op_is_a_constant_to_functorch_where_nothing_of_it_is_tracked():
    def loss(factor):
        op(*arguments("meta"))
        with torch.no_grad():
            call = arguments("meta")
            call[0] = call[0] * factor
            op(*call)
        return factor * 2

    assert torch.func.grad(loss)(torch.ones((), device="meta")).shape == ()


def test_op_writes_outputs_made_in_inference_mode():
    call = arguments("meta")
    with torch.inference_mode():
        call[12] = torch.empty_like(call[0])
    op(*call)                                    # outside of inference mode
    with torch.inference_mode():
        op(*call)
    normal = arguments("meta")
    op(*normal)
    assert normal[12]._version == 1


@pytest.mark.parametrize("device", ["cpu", "meta"])
def test_tensors_elsewhere_get_the_front_ends_error(device):
    """Also once the native side is connected, and on a machine without a device."""
    host.connect()
    with pytest.raises(CompileError, match="CUDA tensor"):
        ops.sparse_mla(*arguments(device))
    i32 = lambda *shape: torch.empty(shape, dtype=torch.int32, device=device)  # noqa: E731
    for ratio in (1, 2, 1 << 70):
        with pytest.raises(CompileError, match="CUDA tensor"):
            neighbours.topk_indices(torch.empty((2, 8), device=device), i32(2), i32(1), i32(1), ratio=ratio)
    rows, cache = (torch.empty(shape, dtype=torch.bfloat16, device=device) for shape in ((2, 512), (2, 128, 1, 512)))
    with pytest.raises(CompileError, match="CUDA tensors"):
        neighbours.cache_append(rows, cache, i32(1, 2), i32(2), i32(1))


def test_package_imports_and_traces_where_the_native_module_cannot_be_built(tmp_path):
    """A copy of the package on a machine with no compiler and nothing built: as with a torch without CUDA."""
    import os
    import shutil
    import subprocess
    import sys
    from pathlib import Path

    root = Path(__file__).resolve().parents[1]
    shutil.copytree(root / "ascendflow_b200", tmp_path / "ascendflow_b200", ignore=shutil.ignore_patterns("lib", "__pycache__"))
    shutil.copytree(root / "include", tmp_path / "include")
    program = """
import torch
from ascendflow_b200 import host, neighbours, ops
from ascendflow_b200.diagnostics import CompileError
shapes = [(4, 64, 512), (8, 128, 1, 512), (8, 64, 1, 512), (4, 1, 512), (2, 3), (2, 3), (3,), (2,), (2,), (2,), (4, 1), (64,), (4, 64, 512)]
types = [torch.bfloat16] * 3 + [torch.int32] * 8 + [torch.float32, torch.bfloat16]
make = lambda device: [torch.empty(s, dtype=t, device=device) for s, t in zip(shapes, types)]
call = make("meta")
torch.ops.ascendflow_b200.sparse_mla(*call)
for function, arguments in ((neighbours.topk_indices, (call[11],) * 4), (neighbours.cache_append, call[:5])):
    try:
        function(*arguments)
    except CompileError:
        continue
    raise SystemExit("not refused")
try:
    host.connect()
except RuntimeError as error:
    assert "not available" in str(error) and error.__cause__ is not None
else:
    raise SystemExit("connected")
print("imported")
"""
    result = subprocess.run([sys.executable, "-c", program], cwd=tmp_path, capture_output=True, text=True,
                            env=dict(os.environ, CXX="/bin/false", PYTHONPATH=str(tmp_path)))
    assert result.stdout.strip().endswith("imported"), result.stderr[-2000:]


def test_host_library_is_identified_by_its_command_and_replaced_as_a_whole(tmp_path, monkeypatch):
    from ascendflow_b200 import build

    identity = build._host_identity()
    monkeypatch.setattr(build, "HOST_FLAGS", ("-O0", *build.HOST_FLAGS[1:]))
    assert build._host_identity() != identity

    library = tmp_path / "_host_calls.so"
    library.write_bytes(b"in use by another rank")
    inode = library.stat().st_ino
    monkeypatch.setattr(build, "HOST_LIBRARY", library)
    monkeypatch.setattr(build, "HOST_STAMP", library.with_suffix(".stamp"))
    monkeypatch.setenv("CXX", str(tmp_path / "compiler"))
    (tmp_path / "compiler").write_text("#!/bin/sh\nwhile [ \"$1\" != -o ]; do shift; done\necho built > \"$2\"\n")
    (tmp_path / "compiler").chmod(0o755)
    with open(library, "rb") as loaded:
        assert build.build_host_library() == library
        assert loaded.read() == b"in use by another rank"   # the file that was there is untouched
    assert library.read_bytes() == b"built\n" and library.stat().st_ino != inode
    assert build.HOST_STAMP.read_text() == build._host_identity()
    assert sorted(path.name for path in tmp_path.iterdir()) == ["_host_calls.so", "_host_calls.stamp", "compiler"]


def test_entry_points_are_handed_over_again_when_the_front_end_comes_last(monkeypatch):
    """A program that selects or appends before it imports the operator: the operator's import clears the entry points, and
    calls went through the Python front end for good, whose reports `ops.status()` does not read."""
    class Recorder:
        def configure(self, *given):
            self.given = given

    recorder, fallback = Recorder(), object()
    monkeypatch.setattr(host, "calls", recorder)
    monkeypatch.setattr(host, "_connected", False)
    monkeypatch.setattr(host, "_fallback", None)
    assert host.connect() and recorder.given[3] is None      # `neighbours` first
    host.set_fallback(fallback)                              # then `ops`
    assert recorder.given == (0, 0, 0, fallback)
    assert host.connect() and all(recorder.given[:3]) and recorder.given[3] is fallback
    assert not host.connect()
