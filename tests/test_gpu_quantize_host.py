"""The native host side of small quantiser calls (csrc/host.cpp) against the general path, which the same call takes without it: same outputs (shapes, strides, types and
bytes), and None - so that the general path runs, with its checks and errors - for everything that is not a plain contiguous CUDA matrix."""
import subprocess
import sys

import pytest
import torch

import sm120fp4_b200 as pkg
from conftest import ROOT
from sm120fp4_b200 import _lib

pytestmark = pytest.mark.gpu


def general(monkeypatch, fn):
    with monkeypatch.context() as m:
        m.setattr(_lib, "_host", _lib.NO_HOST)
        return fn()


def same(a, b):
    assert len(a) == len(b) == 3
    for s, t in zip(a, b):
        assert s.shape == t.shape and s.stride() == t.stride() and s.dtype == t.dtype and s.device == t.device and s.requires_grad == t.requires_grad
        assert torch.equal(s.view(torch.uint8), t.view(torch.uint8))


# 64 x 2048 is the largest matrix that needs no workspace; 65 x 2048 and all matrices beyond take the general path
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,k", [(1, 16), (3, 80), (16, 2048), (64, 2048), (65, 2048), (8192, 16), (129, 1040)])
def test_outputs(monkeypatch, rows, k, dtype):
    x = torch.randn(rows, k, device="cuda", generator=torch.Generator("cuda").manual_seed(rows)).to(dtype).requires_grad_(rows == 3)
    taken = _lib.host().quantize_own_scale(x)
    assert (taken is not None) == (rows * k <= 64 * 2048)
    want = general(monkeypatch, lambda: pkg.quantize_nvfp4(x))
    same(pkg.quantize_nvfp4(x), want)
    gs = want[2]
    assert _lib.host().quantize_128x4(x, gs) is not None
    got = pkg.quantize_nvfp4_128x4(x, gs)
    assert got[2] is gs
    same(got, general(monkeypatch, lambda: pkg.quantize_nvfp4_128x4(x, gs)))


def test_what_is_left_to_the_general_path(monkeypatch):
    h = _lib.host()
    x, gs = torch.randn(8, 64, device="cuda"), torch.ones(1, device="cuda")
    views = [x.t()[:16], x[:, :32], x[::2], x[:0], x[:, :0], x[0], x[None], x.half(), x[:, :24].contiguous(), x.cpu(), torch.nn.Parameter(x), x.to_sparse(), None, 3, "x"]
    for v in views[:10] + views[11:]:
        assert h.quantize_own_scale(v) is None and h.quantize_128x4(v, gs) is None
    for g in (torch.ones((), device="cuda"), torch.ones(2, device="cuda"), torch.ones(1), torch.ones(1, device="cuda", dtype=torch.float64), None, 1.0):
        assert h.quantize_128x4(x, g) is None
    assert torch.vmap(lambda v: (h.quantize_own_scale(v) is None) * v)(torch.randn(2, 8, 64, device="cuda")).sum() != 0   # inside a transform
    from torch.overrides import TorchFunctionMode

    class Seen(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))
    with Seen():
        assert h.quantize_own_scale(x) is None
    for v in (x[:, :32], x[::2], x.half()):       # results and errors are the general path's
        same(pkg.quantize_nvfp4(v), general(monkeypatch, lambda: pkg.quantize_nvfp4(v)))
    with pytest.raises(ValueError):
        pkg.quantize_nvfp4(x[:, :24].contiguous())
    with pytest.raises(TypeError):
        pkg.quantize_nvfp4_128x4(x.half(), gs)
    with pytest.raises(TypeError):
        h.bind(1)


def test_streams_and_capture():
    x = torch.randn(16, 2048, device="cuda", dtype=torch.bfloat16)
    want = [t.clone() for t in pkg.quantize_nvfp4(x)]
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        same(pkg.quantize_nvfp4(x), want)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        out = pkg.quantize_nvfp4(x)
    x.mul_(-1)
    g.replay()
    torch.cuda.synchronize()
    same(out, pkg.quantize_nvfp4(x))


ALLOCATOR = """#include <stddef.h>
int (*held)(void); char* memory; size_t used; int calls, calls_held;
void* take(size_t n, int device, void* stream) { (void)device, (void)stream; ++calls; calls_held += held(); void* p = memory + used; used += n; return p; }
void give(void* p, size_t n, int device, void* stream) { (void)p, (void)n, (void)device, (void)stream; }
"""
ALLOCATE = """
import ctypes, os, sys
import torch
import sm120fp4_b200 as pkg
a = ctypes.CDLL(sys.argv[1])
memory = torch.empty(64 << 20, dtype=torch.uint8, device="cuda")      # (a segment of small blocks is 2 MB, of large ones 20 MB)
x, y, gs = torch.randn(16, 2048, device="cuda"), torch.randn(2048, 2048, device="cuda"), torch.ones(1, device="cuda")
ctypes.c_void_p.in_dll(a, "held").value = ctypes.cast(ctypes.pythonapi.PyGILState_Check, ctypes.c_void_p).value
ctypes.c_void_p.in_dll(a, "memory").value = memory.data_ptr()
calls, held = ctypes.c_int.in_dll(a, "calls"), ctypes.c_int.in_dll(a, "calls_held")
allocator = torch.cuda.memory.CUDAPluggableAllocator(sys.argv[1], "take", "give")
pool = torch.cuda.MemPool(allocator.allocator())
with torch.cuda.use_mem_pool(pool):
    out = pkg.quantize_nvfp4(x)
    first = calls.value
    more = pkg.quantize_nvfp4_128x4(y, gs)
torch.cuda.synchronize()
print(first, calls.value - first, held.value, flush=True)
os._exit(0)      # (the pool's memory is another tensor's: nothing takes it apart)
"""


def test_allocations_leave_the_interpreter_to_other_threads(tmp_path):
    """An allocation that has to wait for the device must not hold the interpreter, which a callback on the device's way may want. An allocator that looks
    whether its caller holds it, and hands out memory that another tensor owns."""
    (tmp_path / "a.c").write_text(ALLOCATOR)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "a.so"), str(tmp_path / "a.c")], check=True)
    r = subprocess.run([sys.executable, "-c", ALLOCATE, str(tmp_path / "a.so")], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    first, second, held = map(int, r.stdout.split())
    assert first > 0 and second > 0 and held == 0
