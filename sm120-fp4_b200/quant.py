"""NVFP4 quantizer on the GPU with the interface of sm120fp4/reference.py (global_scale_for, quantize_nvfp4); results are
bit-identical to the reference's CPU code. `quantize_nvfp4_128x4` is the fused form that writes the block scales
directly in the 128x4 swizzle (optionally gathering source rows), as the W4A4 path consumes them."""
from __future__ import annotations

import torch

from . import _lib
from .layouts import padded_sf_shape

BLOCK = 16


def _dtype_code(x: torch.Tensor) -> int:
    if x.dtype == torch.bfloat16:
        return 0
    if x.dtype == torch.float32:
        return 1
    raise TypeError(f"the quantizer takes bf16 or fp32, not {x.dtype}")


def global_scale_for(x: torch.Tensor) -> torch.Tensor:
    """448 * 6 / amax(|x|) as fp32 [1] (sm120fp4/reference.py:68-71), computed on the device."""
    x = x.contiguous()
    scratch = torch.empty(1, dtype=torch.int32, device=x.device)
    gs = torch.empty(1, dtype=torch.float32, device=x.device)
    _lib.check(_lib.lib().b200moe_global_scale(_lib.ptr(x), _dtype_code(x), x.numel(), _lib.ptr(scratch), _lib.ptr(gs),
                                               _lib.stream_ptr()), "global_scale_for")
    return gs


def _check_2d(x: torch.Tensor) -> None:
    if x.dim() != 2 or x.shape[1] % BLOCK:
        raise ValueError(f"expected [M, K] with K a multiple of {BLOCK}, got {tuple(x.shape)}")
    if not x.is_cuda:
        raise RuntimeError("quantize_nvfp4 runs on the GPU; there is no CPU path in this package")


_ONE_CLUSTER = _lib.ONE_CLUSTER
_WS: dict = {}                # (device index, stream) -> zeroed workspace of eager calls, grown on demand


def _workspace(device: torch.device, stream: int, nbytes: int) -> torch.Tensor:
    """Zeroed once and kept for the eager calls of one stream, which the stream runs one after the other. A captured call is replayed
    on any stream at any later time, and its zeroing runs with the replay: it gets a workspace of its own, from the graph's memory."""
    if torch.cuda.is_current_stream_capturing():
        return torch.zeros(nbytes, dtype=torch.uint8, device=device)
    key = (device.index, stream)
    ws = _WS.get(key)
    if ws is None or ws.numel() < nbytes:
        if len(_WS) >= 64:     # streams come and go: the memory of those of long ago goes back to torch's allocator
            _WS.pop(next(iter(_WS)), None)
        ws = _WS[key] = torch.zeros(max(nbytes, 4096), dtype=torch.uint8, device=device)
    return ws


def _new(rows: int, cols: int, device: torch.device) -> torch.Tensor:
    """An uninitialised uint8 matrix. `empty_strided` takes about half the host time of `empty`, and a small quantiser call is host
    time for the most part."""
    return torch.empty_strided((rows, cols), (cols, 1), dtype=torch.uint8, device=device)


def _own_scale(x: torch.Tensor, groups: int, rows: int, k: int, gs, packed, sf, layout: int, what: str) -> None:
    h = _lib.lib()
    st = _lib.stream_ptr()
    dt = 0 if x.dtype == torch.bfloat16 else 1
    ws, nbytes = None, 0
    if groups > 1 or rows * k > _ONE_CLUSTER:
        nbytes = h.b200moe_quantize_own_scale_workspace_bytes(dt, groups, rows, k)
        ws = _workspace(x.device, st, nbytes)
    rc = h.b200moe_quantize_nvfp4_own_scale(x.data_ptr(), dt, groups, rows, k, gs.data_ptr(), packed.data_ptr(),
                                            sf.data_ptr(), layout, _lib.ptr(ws), nbytes, st)
    if rc:
        _lib.check(rc, what)


def _scale_on(device: torch.device, gs: torch.Tensor) -> torch.Tensor:
    if gs.device == device and gs.dtype == torch.float32 and gs.dim() == 1:
        return gs if gs.shape[0] == 1 else gs.reshape(1)
    return gs.to(device=device, dtype=torch.float32).reshape(1).contiguous()


def quantize_nvfp4(x: torch.Tensor, global_scale: torch.Tensor | None = None):
    """x [M, K] bf16/fp32 -> (packed u8 [M, K/2], sf u8 [M, K/16] E4M3 bits row-major, global_scale f32 [1])
    (sm120fp4/reference.py:74-90)."""
    if global_scale is None and type(x) is torch.Tensor and x.is_cuda:      # a small plain matrix in one native call (csrc/host.cpp), else None
        out = (_lib._host or _lib.host()).quantize_own_scale(x)
        if out is not None:
            return out if type(out) is tuple else _lib.check(out, "quantize_nvfp4")
    _check_2d(x)
    if x.dtype not in (torch.bfloat16, torch.float32):
        x = x.float()
    x = x.contiguous()
    m, k = x.shape
    packed = _new(m, k // 2, x.device)
    sf = _new(m, k // BLOCK, x.device)
    if global_scale is None and m:      # amax, scale and codes in one launch
        gs = torch.empty_strided((1,), (1,), dtype=torch.float32, device=x.device)
        _own_scale(x, 1, m, k, gs, packed, sf, 0, "quantize_nvfp4")
        return packed, sf, gs
    gs = global_scale_for(x) if global_scale is None else _scale_on(x.device, global_scale)
    _lib.check(_lib.lib().b200moe_quantize_nvfp4(_lib.ptr(x), _dtype_code(x), 0, m, k, _lib.ptr(gs), 0, _lib.ptr(packed), _lib.ptr(sf), 0,
                                                 _lib.stream_ptr()), "quantize_nvfp4")
    return packed, sf, gs


def quantize_nvfp4_128x4(x: torch.Tensor, global_scale: torch.Tensor, src_row: torch.Tensor | None = None,
                         out_rows: int | None = None):
    """Fused quantizer: packed u8 [R, K/2] and block scales written directly in the 128x4 swizzle ([pad128(R), pad4(K/16)]).
    With `src_row` (int32 [R]) destination row r reads x[src_row[r]] (negative: a zero row), which lays tokens out in
    per-expert segments without a separate gather."""
    if src_row is None and type(x) is torch.Tensor and x.is_cuda:      # (as in quantize_nvfp4)
        out = (_lib._host or _lib.host()).quantize_128x4(x, global_scale)
        if out is not None:
            return out if type(out) is tuple else _lib.check(out, "quantize_nvfp4_128x4")
    _check_2d(x)
    x = x.contiguous()
    k = x.shape[1]
    rows = x.shape[0] if src_row is None else (int(src_row.numel()) if out_rows is None else out_rows)
    pr, pc = padded_sf_shape(rows, k // BLOCK)
    gs = _scale_on(x.device, global_scale)
    packed = _new(rows, k // 2, x.device)
    sf = _new(pr, pc, x.device)     # the kernel writes the padding too
    if rows == 0:
        sf.zero_()
    if src_row is not None:
        src_row = src_row.to(device=x.device, dtype=torch.int32).contiguous()
    _lib.check(_lib.lib().b200moe_quantize_nvfp4(_lib.ptr(x), _dtype_code(x), _lib.ptr(src_row), rows, k, _lib.ptr(gs), 0, _lib.ptr(packed),
                                                 _lib.ptr(sf), 1, _lib.stream_ptr()), "quantize_nvfp4_128x4")
    return packed, sf, gs


def quantize_nvfp4_experts(w: torch.Tensor, swizzle: bool = False):
    """Stacked expert matrices w [E, R, K] -> (packed u8 [E, R, K/2], sf u8 [E, R, K/16] row-major or [E, pad128(R),
    pad4(K/16)] in the 128x4 swizzle, global_scale f32 [E]): each expert quantised with its own global scale
    2688 / amax, exactly as E separate calls of the reference's quantize_nvfp4 would, in one launch."""
    if w.dim() != 3 or w.shape[2] % BLOCK:
        raise ValueError(f"expected [E, R, K] with K a multiple of {BLOCK}, got {tuple(w.shape)}")
    if not w.is_cuda:
        raise RuntimeError("quantize_nvfp4_experts runs on the GPU; there is no CPU path in this package")
    w = w.contiguous()
    e, r, k = w.shape
    if w.dtype not in (torch.bfloat16, torch.float32):
        _dtype_code(w)                       # raises
    gs = torch.empty(e, dtype=torch.float32, device=w.device)
    packed = torch.empty((e, r, k // 2), dtype=torch.uint8, device=w.device)
    pr, pc = padded_sf_shape(r, k // BLOCK) if swizzle else (r, k // BLOCK)
    sf = torch.empty((e, pr, pc), dtype=torch.uint8, device=w.device)
    _own_scale(w, e, r, k, gs, packed, sf, 1 if swizzle else 0, "quantize_nvfp4_experts")
    return packed, sf, gs
