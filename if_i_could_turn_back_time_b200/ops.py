"""Operators over packed weights: thin, checked calls into libjq.so.

Everything here runs on the GPU through the C ABI; there is no eager or CPU
fallback.  The fused linear is also registered as ``torch.ops.jq.linear`` so
that it composes with torch's dispatcher (fake tensors, export).
"""
from __future__ import annotations

import ctypes
import threading
import warnings
from typing import List, Optional, Sequence

import numpy as np
import torch

from . import _lib
from .pack import PackedWeight

_DT = {torch.float32: _lib.JQ_F32, torch.float16: _lib.JQ_F16, torch.bfloat16: _lib.JQ_BF16}
MAX_GEMV_BATCH = 8


def _ptr(t: Optional[torch.Tensor]):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def _stream() -> int:
    """Handle of the current device's current stream."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _addr(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


def _need_cuda(*ts):
    for t in ts:
        if t is not None and not t.is_cuda:
            raise RuntimeError("libjq operators run on CUDA tensors only (there is no CPU path)")


def dequantize(pw: PackedWeight) -> torch.Tensor:
    """Dense fp32 [N, K] of a packed matrix (bit-exact definition of W_hat)."""
    lib = _lib.load()
    _need_cuda(pw.qweight, pw.scales, pw.codebook)
    out = torch.empty((pw.N, pw.K), dtype=torch.float32, device=pw.qweight.device)
    with torch.cuda.device(out.device):
        if pw.spec.fmt == "e2m1":
            st = lib.jq_dequant_e2m1(_ptr(pw.qweight), _ptr(pw.scales), _ptr(out), pw.N, pw.K, pw.spec.group_size,
                                     _stream())
        else:
            st = lib.jq_dequant_gf4(_ptr(pw.qweight), _ptr(pw.scales), _ptr(pw.codebook), _ptr(out), pw.N, pw.K,
                                    pw.spec.group_size, _stream())
    _lib.check(st, "jq_dequant")
    return out


def fwht_block(x: torch.Tensor, block: int = 128) -> torch.Tensor:
    """fp32 block Hadamard rotation along the last dim."""
    lib = _lib.load()
    _need_cuda(x)
    x2 = x.reshape(-1, x.shape[-1]).contiguous()
    y = torch.empty(x2.shape, dtype=torch.float32, device=x.device)
    with torch.cuda.device(x.device):
        st = lib.jq_fwht_block(_ptr(x2), _ptr(y), x2.shape[0], x2.shape[1], block, _DT[x2.dtype], _stream())
    _lib.check(st, "jq_fwht_block")
    return y.reshape(x.shape)


_OUT = {-1: None, _lib.JQ_F32: torch.float32, _lib.JQ_F16: torch.float16, _lib.JQ_BF16: torch.bfloat16}


def ta_max_batch(fmt_id: int) -> int:
    """Rows one pass of the pair-table / tensor-memory kernels takes."""
    return 64


def ta_eligible(fmt_id: int, K: int, g: int, batch: int) -> bool:
    """Problems the TMA-fed kernels take.  GF4 (group size 128 * 2^k): every
    batch -- one row (while the prepared activation fits in shared memory, K
    up to 12288) on the CUDA-core pair-table loop, the rest on the
    tensor-memory kernel.  E2M1 g32: batches from 9 rows on the tensor-memory
    kernel (up to 8 rows the mma.sync row loops are faster).  64 rows per
    pass."""
    if K % 256 or K < 512:
        return False
    if fmt_id == _lib.JQ_FMT_GF4:
        gq = g >> 7
        return g >= 128 and g % 128 == 0 and gq & (gq - 1) == 0 and K % g == 0 and batch >= 1
    return g == 32 and batch >= 9


def _ta_aligned(*tensors) -> bool:
    """The TMA-fed kernels read E2M1 scales in 16-byte pieces (the row loops in 2- or 4-byte pieces); a view that
    starts elsewhere is served by the row loops instead.  Packed rows and codebooks are 16-byte aligned on every
    path (the library refuses anything else)."""
    return all(t is None or t.data_ptr() % 16 == 0 for t in tensors)


MAX_ROWS_SCRATCH = 256 << 20      # bytes of prepared activation a many-row call holds at once; longer inputs go in parts


def many_rows(fmt_id: int, K: int, g: int, batch: int) -> bool:
    """Calls that the many-row kernel takes: more rows than the kernels for small batches take well.  Those read the
    weights once per pass (8 rows for the shapes that only the row loops take, which keep 9 to 16 rows, two passes), the
    many-row kernel decodes them once per 256 rows.

    GF4 on the tensor-memory kernel's shapes: up to 32 rows that kernel is the faster one everywhere, from 33 rows it
    depends on the matrix, as it no longer splits a row over CTAs.  Device time of a call in us, tensor-memory kernel /
    many-row kernel (two to four passes of 16 rows, the only kernel there was before):

        rows   1024 x 1024           4096 x 4096           11008 x 4096          4096 x 11008          28672 x 8192
        17     10.5 / 11.6 (16.1)    13.6 / 20.6 (29.8)    22.0 / 40.4 (35.9)    22.5 / 43.0 (61.4)    75.7 / 142 (119)
        32     10.5 / 11.7 (18.9)    15.0 / 20.5 (37.8)    22.1 / 40.9 (38.0)    25.0 / 43.1 (83.6)    76.9 / 142 (130)
        48     11.8 / 11.8 (28.0)    23.3 / 24.4 (56.5)    23.8 / 41.4 (57.0)    52.5 / 46.1 (125)     81.1 / 144 (196)
        64     12.3 / 12.1 (37.5)    23.3 / 24.5 (75.5)    25.7 / 41.6 (75.7)    52.8 / 46.2 (167)     81.6 / 144 (260)"""
    if ta_eligible(fmt_id, K, g, batch):
        return batch > (32 if fmt_id == _lib.JQ_FMT_GF4 else ta_max_batch(fmt_id))
    return batch > 16


# Smallest scratch buffer of a kernel family, 1 MB if not named here.  "ta": one pass of 64 rows of up to 32000 codes, so that calls on a stream
# that has made one, in a graph capture too, do not need a larger one.
_LEAST_SCRATCH = {"ta": 4 << 20}
_tls = threading.local()   # every host thread has its own scratch buffers: calls from different threads never share one
_captured = {}             # address -> buffer that a graph capture has used: the graph replays into it, so it is never freed
_checked = False


def _ws_cache() -> dict:
    d = getattr(_tls, "ws", None)
    if d is None:
        d = _tls.ws = {}
    return d


def set_checked(on: bool) -> None:
    """Checked mode: every call that runs a kernel with device-side waits (the
    pair-table and tensor-memory kernels) is followed by a read of its status
    word, which synchronises the stream, and raises if a wait gave up.  Off by
    default: the status stays in the workspace until ``check_status()``."""
    global _checked
    _checked = bool(on)


def _capturing(stream: int) -> bool:
    """Whether a graph is being captured on the current stream.  The legacy default stream (0) cannot be captured, and
    calls on it save the 0.4 us that asking takes."""
    return stream != 0 and torch.cuda.is_current_stream_capturing()


def _workspace(device, nbytes: int, kind: str = "gemv") -> torch.Tensor:
    """Grow-only scratch per (device, stream, kernel family): calls on one
    stream are ordered, so consecutive calls may share it; another stream gets
    its own.  The family with a status word at offset 0 ("ta") never shares
    a buffer with the split-K partial sums, and starts zeroed.  A buffer that a
    captured call has used stays alive when a larger one takes its place or its
    thread ends; the successor is at least twice as large, so that what a
    stream keeps is at most its newest buffer's size."""
    index = torch._C._cuda_getDevice() if device.index is None else device.index
    key = (index, torch._C._cuda_getCurrentRawStream(index), kind)
    cache = _ws_cache()
    t = cache.get(key)
    if t is None or t.numel() < nbytes:
        if t is not None and kind != "gemv" and check_status(raise_on_error=False):
            raise RuntimeError("a device-side wait gave up in an earlier call (status word raised)")
        least = 2 * t.numel() if t is not None and t.data_ptr() in _captured else _LEAST_SCRATCH.get(kind, 1 << 20)
        t = torch.zeros(max(nbytes, least), dtype=torch.uint8, device=device)
        cache[key] = t
    if _capturing(key[1]):
        _captured[t.data_ptr()] = t
    return t


def reserve_workspace(device, nbytes: int, kind: str = "ta") -> None:
    """Allocate this thread's scratch for (device, current stream, kernel family) ahead of time, e.g. before a
    CUDA-graph capture or a region that must not allocate: kind "gemv" = split-K partial sums of the row loops,
    "ta" = prepared activations and status word of the TMA-fed kernels."""
    _workspace(torch.device(device), nbytes, kind)


def check_status(raise_on_error: bool = True) -> int:
    """Read and clear the sticky status words of this device's workspaces on
    the current stream (synchronises).  A kernel whose bounded wait expired
    leaves JQ_ERR_TIMEOUT there and returns early with its outputs partly
    written; every later call keeps the word until it is read here."""
    lib = _lib.load()
    worst = 0
    ws = _ws_cache().get((torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream, "ta"))
    if ws is not None:
        worst = min(worst, lib.jq_ta_status(_ptr(ws), 1, _stream()))
    if worst and raise_on_error:
        raise _lib.JqError(worst, "device status")
    return worst


_ta_workspace_bytes = {}       # (K, rows) -> bytes


def _linear_rows_ta(x2, qweight, scales, codebook, bias, fmt_id, N, K, g, had, y):
    """Through the TMA-fed kernels, at most ta_max_batch rows per pass."""
    lib = _lib.load()
    Bt = x2.shape[0]
    most = ta_max_batch(fmt_id)
    with _on(x2.device):
        stream = _stream()
        for b0 in range(0, Bt, most):
            b1 = min(Bt, b0 + most)
            wsb = _ta_workspace_bytes.get((K, b1 - b0))
            if wsb is None:
                prob = _lib.jq_problem()
                prob.K = K
                wsb = _ta_workspace_bytes[(K, b1 - b0)] = lib.jq_ta_workspace_bytes(ctypes.byref(prob), 1, b1 - b0)
            ws = _workspace(x2.device, wsb, "ta")
            xs, ys = (x2, y) if Bt <= most else (x2[b0:b1], y[b0:b1])
            st = lib.jq_gemm_ta(fmt_id, _addr(qweight), _addr(scales), _addr(codebook), xs.data_ptr(), _addr(bias),
                                ys.data_ptr(), N, K, b1 - b0, g, had, _DT[x2.dtype], _DT[y.dtype], ws.data_ptr(), ws.numel(),
                                stream)
            if st:
                _lib.check(st, "jq_gemm_ta")
    if _checked:
        check_status()
    return y


def _rows_scratch(device, nbytes: int):
    """(scratch pointer, size, status word) of a many-row call: the thread's "ta" buffer when the prepared activation
    fits into it as it is, an allocation of the call's own otherwise, and always while a graph is captured (from the
    graph's pool: graphs that were captured on one stream may replay on several).  The status word is the buffer's."""
    ws = _workspace(device, 1024, "ta")
    if ws.numel() >= 1024 + nbytes and not _capturing(_stream()):
        return None, ws.data_ptr() + 1024, ws.numel() - 1024, ws.data_ptr()
    own = torch.empty(nbytes, dtype=torch.uint8, device=device)
    return own, own.data_ptr(), nbytes, ws.data_ptr()


_rows_scratch_bytes = {}       # (device, format, N, K, rows, group size) -> bytes


def _many_rows_scratch_bytes(lib, *key) -> int:
    """Scratch of a many-row call on the current device; the library searches for the call's tile shape to know it."""
    key = (torch._C._cuda_getDevice(), *key)
    n = _rows_scratch_bytes.get(key)
    if n is None:
        if len(_rows_scratch_bytes) >= 4096:
            _rows_scratch_bytes.clear()
        n = _rows_scratch_bytes[key] = lib.jq_gemm_rows_scratch_bytes(*key[1:])
    return n


def _linear_many_rows(x2, qweight, scales, codebook, bias, fmt_id, N, K, g, had, y):
    lib = _lib.load()
    rows = x2.shape[0]
    part = max(256, MAX_ROWS_SCRATCH // ((K + 127) // 128 * 256) // 256 * 256)
    with _on(x2.device):
        for b0 in range(0, rows, part):
            b1 = min(rows, b0 + part)
            xs, ys = (x2, y) if rows <= part else (x2[b0:b1], y[b0:b1])
            own, scratch, size, status = _rows_scratch(x2.device, _many_rows_scratch_bytes(lib, fmt_id, N, K, b1 - b0, g))
            st = lib.jq_gemm_rows(fmt_id, _addr(qweight), _addr(scales), _addr(codebook), xs.data_ptr(), _addr(bias),
                                  ys.data_ptr(), N, K, b1 - b0, g, had, _DT[x2.dtype], _DT[y.dtype], scratch, size, status,
                                  _stream())
            if st:
                _lib.check(st, "jq_gemm_rows")
            del own
    if _checked:
        check_status()
    return y


_Strides = ctypes.c_int64 * 4


def conv2d(x: torch.Tensor, pw: PackedWeight, bias: Optional[torch.Tensor], kernel_size, stride, padding,
           dilation) -> torch.Tensor:
    """The receptive fields of x [B, C, H, W] times the packed [O, C*kh*kw] matrix -> [B, O, ho, wo] (channels-last
    strides): the fields are gathered by the preparation kernel, there is no unfolded copy."""
    if x.dim() != 4:
        raise RuntimeError(f"x has {x.dim()} dimensions, a convolution takes [B, C, H, W]")
    if x.dtype not in _DT:
        raise RuntimeError(f"unsupported activation dtype {x.dtype}")
    B, C, H, W = x.shape
    geo = [int(v) for pair in (kernel_size, stride, padding, dilation) for v in pair]
    kh, kw, stride_h, stride_w, pad_h, pad_w, dil_h, dil_w = geo
    if C * kh * kw != pw.K:
        raise RuntimeError(f"x has {C} channels: fields of {C * kh * kw} values, packed weight has K={pw.K}")
    if pw.spec.had_block:
        raise RuntimeError("a rotated weight needs the fields laid out for the linear operator")
    ho = (H + 2 * pad_h - dil_h * (kh - 1) - 1) // stride_h + 1
    wo = (W + 2 * pad_w - dil_w * (kw - 1) - 1) // stride_w + 1
    if ho <= 0 or wo <= 0:
        raise RuntimeError(f"an image of {H} x {W} leaves no output position")
    lib = _lib.load()
    _need_cuda(x, pw.qweight, pw.scales, pw.codebook, bias)
    if bias is not None and bias.dtype != torch.float32:
        bias = bias.float()
    x = x.resolve_neg()        # (the imaginary part of a conjugate is a view whose sign is not in memory)
    L = ho * wo
    y = torch.empty((B * L, pw.N), dtype=x.dtype, device=x.device)
    part = max(1, MAX_ROWS_SCRATCH // ((pw.K + 127) // 128 * 256) // L)          # images at once
    with _on(x.device):
        for b0 in range(0, B, part):
            b1 = min(B, b0 + part)
            rows, fmt_id, g = (b1 - b0) * L, pw.spec.fmt_id, pw.spec.group_size
            xs, ys = (x, y) if b1 - b0 == B else (x[b0:b1], y[b0 * L:b1 * L])
            c = _lib.jq_conv(b1 - b0, C, H, W, *geo, _Strides(*x.stride()))
            own, scratch, size, status = _rows_scratch(x.device, _many_rows_scratch_bytes(lib, fmt_id, pw.N, pw.K, rows, g))
            st = lib.jq_conv_rows(fmt_id, _addr(pw.qweight), _addr(pw.scales), _addr(pw.codebook), xs.data_ptr(), _addr(bias),
                                  ys.data_ptr(), ctypes.byref(c), pw.N, pw.K, rows, g, _DT[x.dtype], _DT[y.dtype], scratch, size,
                                  status, _stream())
            if st:
                _lib.check(st, "jq_conv_rows")
            del own
    if _checked:
        check_status()
    return y.view(B, ho, wo, pw.N).permute(0, 3, 1, 2)


def conv_gathers(fmt_id: int, K: int, g: int, positions: int) -> bool:
    """Convolutions whose fields the preparation kernel gathers (the others are unfolded first): the output positions that
    the many-row kernel is for, and fields of up to 1536 values or more than 2048 positions.  A block gathers 32 positions and
    walks along the whole field, so that long fields at few positions leave most of the chip idle.

    The line of 2048 positions was drawn when the gathering formed its addresses by products and took two to three times as
    long.  Where it lies now, calls of 1024 to 2048 positions with more than 1536 values are still unfolded although gathering
    would be faster, and so are 784 positions of 2304 values.  Whole calls of a layer with 3 x 3 kernels and 256 outputs, us,
    gathered / unfolded (784 positions: four images, 1024 and 2048: images of 16 x 16 and 32 x 32):

        positions   K = 2304       K = 4608       K = 9216
        196         36 / 53        60 / 52        107 / 57
        784         42 / 52        66 / 67        112 / 107
        1024        56 / 89        81 / 103       130 / 157
        1568        46 / 116       70 / 137       117 / 222
        2048        46 / 80        72 / 130       142 / 250
        3136        52 / 124       77 / 197       129 / 355

    On the device alone 196 positions of 2304 values take 33 / 26, and of 1152 values 22 / 21."""
    few = ta_max_batch(fmt_id) if fmt_id == _lib.JQ_FMT_E2M1 and ta_eligible(fmt_id, K, g, positions) else 16
    return positions > few and (K <= 1536 or positions > 2048)


_wsb_cache = {}


class _NoDeviceSwitch:
    def __enter__(self):
        return None

    def __exit__(self, *exc):
        return False


_NO_SWITCH = _NoDeviceSwitch()


def _on(device):
    """Device guard that costs nothing when the tensor's device is already current."""
    return _NO_SWITCH if device.index == torch._C._cuda_getDevice() else torch.cuda.device(device)


def _linear_rows(x2, qweight, scales, codebook, bias, fmt_id, N, K, g, had, out_id=-1):
    lib = _lib.load()
    Bt = x2.shape[0]
    y = torch.empty((Bt, N), dtype=_OUT[out_id] or x2.dtype, device=x2.device)
    if many_rows(fmt_id, K, g, Bt):
        return _linear_many_rows(x2, qweight, scales, codebook, bias, fmt_id, N, K, g, had, y)
    if ta_eligible(fmt_id, K, g, Bt):
        if _ta_aligned(qweight, scales, codebook):
            return _linear_rows_ta(x2, qweight, scales, codebook, bias, fmt_id, N, K, g, had, y)
        if fmt_id == _lib.JQ_FMT_GF4 and Bt > 16:       # scales off a 16-byte boundary, which the many-row kernel takes
            return _linear_many_rows(x2, qweight, scales, codebook, bias, fmt_id, N, K, g, had, y)
    xd, yd = _DT[x2.dtype], _DT[y.dtype]
    qw_p, sc_p, cb_p, bias_p = _addr(qweight), _addr(scales), _addr(codebook), _addr(bias)
    with _on(x2.device):
        stream = _stream()
        for b0 in range(0, Bt, MAX_GEMV_BATCH):
            b1 = min(Bt, b0 + MAX_GEMV_BATCH)
            xs, ys = (x2, y) if Bt <= MAX_GEMV_BATCH else (x2[b0:b1], y[b0:b1])
            # split-K scratch (fp32 partial outputs) when the staged batch would not fit in shared memory
            key = (N, K, b1 - b0)
            wsb = _wsb_cache.get(key)
            if wsb is None:
                wsb = _wsb_cache[key] = lib.jq_workspace_bytes(0, N, K, b1 - b0)
            ws = _workspace(x2.device, wsb)[:wsb] if wsb else None

            def call(ws_t):
                nb = ws_t.numel() if ws_t is not None else 0
                if fmt_id == _lib.JQ_FMT_E2M1:
                    return lib.jq_gemv_e2m1(qw_p, sc_p, xs.data_ptr(), bias_p, ys.data_ptr(), N, K,
                                            b1 - b0, g, had, xd, yd, _addr(ws_t), nb, stream)
                return lib.jq_gemv_gf4(qw_p, sc_p, cb_p, xs.data_ptr(), bias_p, ys.data_ptr(),
                                       N, K, b1 - b0, g, had, xd, yd, _addr(ws_t), nb, stream)

            st = call(ws)
            if st == -6 and ws is not None:   # workspace too small for this group size: sub-batch path
                st = call(None)
            if st:
                _lib.check(st, "jq_gemv")
    return y


@torch.library.custom_op("jq::linear", mutates_args=(), device_types="cuda")
def _jq_linear(x: torch.Tensor, qweight: torch.Tensor, scales: Optional[torch.Tensor],
               codebook: Optional[torch.Tensor], bias: Optional[torch.Tensor], fmt_id: int, N: int, K: int,
               group_size: int, had_block: int, out_id: int) -> torch.Tensor:
    x2 = x.reshape(-1, K).contiguous()
    y = _linear_rows(x2, qweight, scales, codebook, bias, fmt_id, N, K, group_size, had_block, out_id)
    return y.reshape(*x.shape[:-1], N)


@_jq_linear.register_fake
def _(x, qweight, scales, codebook, bias, fmt_id, N, K, group_size, had_block, out_id):
    return x.new_empty((*x.shape[:-1], N), dtype=_OUT[out_id] or x.dtype)


def linear(x: torch.Tensor, pw: PackedWeight, bias: Optional[torch.Tensor] = None,
           out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """``F.linear(rotate(x), W_hat, bias)`` without materialising W_hat; any
    leading dims, last dim = K; output dtype = input dtype unless given."""
    if x.shape[-1] != pw.K:
        raise RuntimeError(f"last dim of x is {x.shape[-1]}, packed weight has K={pw.K}")
    if x.dtype not in _DT:
        raise RuntimeError(f"unsupported activation dtype {x.dtype}")
    _need_cuda(x, pw.qweight, pw.scales, pw.codebook, bias)
    if bias is not None and bias.dtype != torch.float32:
        bias = bias.float()
    out_id = -1 if out_dtype is None else _DT[out_dtype]
    if torch.compiler.is_compiling():
        # through the dispatcher so that tracing sees one opaque op with a fake implementation
        return torch.ops.jq.linear(x, pw.qweight, pw.scales, pw.codebook, bias, pw.spec.fmt_id, pw.N, pw.K,
                                   pw.spec.group_size, pw.spec.had_block, out_id)
    flat = x.dim() == 2
    x2 = x if flat else x.reshape(-1, pw.K)
    if not x2.is_contiguous():
        x2 = x2.contiguous()
    y = _linear_rows(x2, pw.qweight, pw.scales, pw.codebook, bias, pw.spec.fmt_id, pw.N, pw.K, pw.spec.group_size,
                     pw.spec.had_block, out_id)
    return y if flat else y.reshape(*x.shape[:-1], pw.N)


class GroupedGemv:
    """A fixed set of independent GEMVs (one decode step's matrices) run in a
    single launch.  Inputs and outputs are preallocated; ``run()`` only
    enqueues the kernel.

    Row-sharded use (one process per GPU): pass each matrix's local shard in
    ``weights``, its unsharded row count in ``full_rows`` and the shard's
    first row in ``row_offsets``; outputs are then full-width ``[batch,
    full_rows]`` buffers of which this rank fills its columns.  With
    ``group`` (a ``torch.distributed`` process group, world size <= 8) the
    output arena lives in symmetric memory and the kernel's epilogue stores
    every result into all ranks' arenas (the all-gather fused into the GEMV);
    call ``barrier()`` after ``run()`` before reading."""

    def __init__(self, weights: Sequence[PackedWeight], batch: int, x_dtype=torch.bfloat16,
                 biases: Optional[Sequence[Optional[torch.Tensor]]] = None, device=None,
                 full_rows: Optional[Sequence[int]] = None, row_offsets: Optional[Sequence[int]] = None,
                 group=None):
        lib = _lib.load()
        if not weights:
            raise ValueError("no problems")
        spec0 = weights[0].spec
        for w in weights:
            if w.spec.fmt != spec0.fmt:
                raise ValueError("a grouped launch needs one weight format")
        self.device = device or weights[0].qweight.device
        self.weights = list(weights)
        self.batch = batch
        self.x_dtype = x_dtype
        self.biases = list(biases) if biases is not None else [None] * len(weights)
        self.full_rows = list(full_rows) if full_rows is not None else [w.N for w in weights]
        self.row_offsets = list(row_offsets) if row_offsets is not None else [0] * len(weights)
        # all inputs live in one arena and all outputs in another, so a step's
        # activations move with one copy each way; every view is 256-byte aligned
        esz = torch.empty((), dtype=x_dtype).element_size()
        rnd = lambda nbytes: (nbytes + 255) // 256 * 256
        x_off, y_off, xo, yo = [], [], 0, 0
        for w, nf in zip(weights, self.full_rows):
            x_off.append(xo); xo += rnd(batch * w.K * esz)
            y_off.append(yo); yo += rnd(batch * nf * esz)
        self.x_arena = torch.zeros(xo, dtype=torch.uint8, device=self.device)
        self._symm = None
        self._peer_delta = np.zeros(1, dtype=np.int64)
        if group is not None and torch.distributed.get_world_size(group) > 1:
            import torch.distributed._symmetric_memory as symm_mem
            self.y_arena = symm_mem.empty(yo, dtype=torch.uint8, device=self.device)
            self.y_arena.zero_()
            self._symm = symm_mem.rendezvous(self.y_arena, group.group_name if hasattr(group, "group_name") else group)
            own = self.y_arena.data_ptr()
            ptrs = [int(p) for p in self._symm.buffer_ptrs]
            if len(ptrs) > 8:
                raise ValueError("at most 8 peers")
            self._peer_delta = np.array([p - own for p in ptrs], dtype=np.int64)
        else:
            self.y_arena = torch.zeros(yo, dtype=torch.uint8, device=self.device)
        self.x_offsets, self.y_offsets = x_off, y_off
        self.xs: List[torch.Tensor] = [
            self.x_arena[o:o + batch * w.K * esz].view(x_dtype).view(batch, w.K) for o, w in zip(x_off, weights)]
        self.ys: List[torch.Tensor] = [
            self.y_arena[o:o + batch * nf * esz].view(x_dtype).view(batch, nf) for o, nf in zip(y_off, self.full_rows)]
        n = len(weights)
        arr = (_lib.jq_problem * n)()
        for i, w in enumerate(weights):
            arr[i].qweight = w.qweight.data_ptr()
            arr[i].scales = w.scales.data_ptr() if w.scales is not None else None
            arr[i].codebook = w.codebook.data_ptr() if w.codebook is not None else None
            arr[i].x = self.xs[i].data_ptr()
            arr[i].bias = self.biases[i].data_ptr() if self.biases[i] is not None else None
            arr[i].y = self.ys[i].data_ptr() + self.row_offsets[i] * esz
            arr[i].N, arr[i].K, arr[i].g, arr[i].had_block = w.N, w.K, w.spec.group_size, w.spec.had_block
            arr[i].ldy = self.full_rows[i]
        self._problems_host = arr
        self._per_problem = False
        self._subs = []
        self._ta = []
        use_ta = all(ta_eligible(w.spec.fmt_id, w.K, w.spec.group_size, batch)
                     and _ta_aligned(w.qweight, w.scales, w.codebook) for w in weights)
        if use_ta:
            MAX_TA_BATCH = ta_max_batch(spec0.fmt_id)
            # through the TMA-fed kernels: one plan (and workspace) per sub-batch of at most 64 rows;
            # a run is one activation-preparation launch plus one persistent launch per sub-batch
            with torch.cuda.device(self.device):
                for b0 in range(0, batch, MAX_TA_BATCH):
                    nb = min(MAX_TA_BATCH, batch - b0)
                    sub = (_lib.jq_problem * n)()
                    ctypes.memmove(sub, arr, ctypes.sizeof(arr))
                    for i, (w, nf) in enumerate(zip(weights, self.full_rows)):
                        sub[i].x = arr[i].x + b0 * w.K * esz
                        sub[i].y = arr[i].y + b0 * nf * esz
                    wsb = lib.jq_ta_workspace_bytes(ctypes.byref(sub), n, nb)
                    ws = torch.zeros(wsb, dtype=torch.uint8, device=self.device)
                    plan_host = np.zeros((lib.jq_ta_plan_bytes(n) + 3) // 4, dtype=np.int32)
                    _lib.check(lib.jq_ta_plan(spec0.fmt_id, ctypes.byref(sub), n, nb, _ptr(ws), wsb,
                                              plan_host.ctypes.data, plan_host.nbytes), "jq_ta_plan")
                    self._ta.append((plan_host, torch.from_numpy(plan_host).to(self.device), ws))
            self.launches_per_run = 2 * len(self._ta)
            return
        # one grouped launch per sub-batch of at most 8 rows (the row loops' limit)
        with torch.cuda.device(self.device):
            for b0 in range(0, batch, MAX_GEMV_BATCH):
                nb = min(MAX_GEMV_BATCH, batch - b0)
                sub = (_lib.jq_problem * n)()
                ctypes.memmove(sub, arr, ctypes.sizeof(arr))
                for i, (w, nf) in enumerate(zip(weights, self.full_rows)):
                    sub[i].x = arr[i].x + b0 * w.K * esz
                    sub[i].y = arr[i].y + b0 * nf * esz
                nbytes = lib.jq_grouped_plan_bytes(n)
                plan_host = np.zeros((nbytes + 3) // 4, dtype=np.int32)
                _lib.check(lib.jq_grouped_plan(spec0.fmt_id, ctypes.byref(sub), n, nb, plan_host.ctypes.data,
                                               plan_host.nbytes), "jq_grouped_plan")
                raw = np.frombuffer(bytes(sub), dtype=np.uint8).copy()
                self._subs.append((torch.from_numpy(raw).to(self.device), plan_host,
                                   torch.from_numpy(plan_host).to(self.device)))
        self.launches_per_run = len(self._subs)

    @property
    def fused_exchange(self) -> bool:
        return self._symm is not None

    def barrier(self) -> None:
        """Order the ranks after run(): every rank's stores into this rank's
        output arena are complete once this returns on the stream."""
        if self._symm is not None:
            self._symm.barrier()

    def status(self, clear: bool = True) -> int:
        """Sticky device status of the pair-table kernels' workspaces (0 = fine);
        synchronises the stream."""
        lib = _lib.load()
        worst = 0
        with torch.cuda.device(self.device):
            for _, _, ws in self._ta:
                worst = min(worst, lib.jq_ta_status(_ptr(ws), 1 if clear else 0, _stream()))
        return worst

    def run(self) -> None:
        lib = _lib.load()
        if self._ta:
            with torch.cuda.device(self.device):
                for plan_host, plan_dev, ws in self._ta:
                    st = lib.jq_gemm_ta_grouped(plan_host.ctypes.data, _ptr(plan_dev), _ptr(ws), _DT[self.x_dtype],
                                                _DT[self.x_dtype], len(self._peer_delta), self._peer_delta.ctypes.data,
                                                _stream())
                    _lib.check(st, "jq_gemm_ta_grouped")
            return
        if not self._per_problem:
            st = 0
            with torch.cuda.device(self.device):
                for problems_dev, plan_host, plan_dev in self._subs:
                    st = lib.jq_gemv_grouped_peers(_ptr(problems_dev), plan_host.ctypes.data, _ptr(plan_dev),
                                                   _DT[self.x_dtype], _DT[self.x_dtype], len(self._peer_delta),
                                                   self._peer_delta.ctypes.data, _stream())
                    if st:
                        break
            if st != -5:
                _lib.check(st, "jq_gemv_grouped")
                return
            if self._symm is not None:
                _lib.check(st, "jq_gemv_grouped_peers")
            # batch x K too large for one staged activation per CTA: one (split-K) launch per matrix instead
            warnings.warn("GroupedGemv: this batch x K does not fit a grouped launch; running one launch per matrix")
            self._per_problem = True
        for w, x, y, b, nf, ro in zip(self.weights, self.xs, self.ys, self.biases, self.full_rows, self.row_offsets):
            y[:, ro:ro + w.N].copy_(linear(x, w, b))
        self.launches_per_run = None
