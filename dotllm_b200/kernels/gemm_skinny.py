"""Dispatch to the weight-streaming products for steps of a few rows (decode).

Up to ``SKINNY_ROWS`` rows go to the mma.sync kernel of csrc/gemm_skinny.cu (it can take 16), more, up
to 128, to the tcgen05 kernel of csrc/gemm_decode_tc.cu (``gemm_decode_tc.run``, same contract).  The first gives every multiprocessor
the same rows of W, or (few sizes) cuts its work into equal shares per warp, where tiles that straddle two shares are summed through a
scratch buffer with arrival counters (``plan`` tells).  Both are kept here per device (they are small and every launch leaves the
counters zero).  Launches that share them must be on one stream.
"""
from __future__ import annotations

import ctypes
import functools

import torch

from . import gemm_decode_tc
from . import library as _library

_P, _I, _F = _library._P, _library._I, _library._F
_library.register_signatures({
    "dl_gemm_skinny_bf16": [_P, _I, _P, _P, _I, _I, _I, _I, _I, _I, _P, _I, _P, _I, _P, _P],
    "dl_gemm_skinny_fused_bf16": [_P, _I, _P, _P, _I, _I, _I, _I, _I, _I, _P, _P, _I, _P, _P, _I, _F, _F,
                                  _P, _I, _P, _I, _P, _P],
    "dl_gemm_skinny_gated_bf16": [_P, _I, _P, _P, _I, _I, _I, _I, _I, _I, _I, _F, _F, _P, _P, _I, _P, _I, _P, _P],
    "dl_gemm_skinny_parts": [_I, _I],
    "dl_gemm_skinny_plan": [_I, _I, _I, _I, _P, _P, _P, _P],
    "dl_gemm_skinny_scratch": [_I, _I, _I, _I, _I, _P, _P],
})

KERNEL_ROWS = 16         # rows the mma.sync kernel can take (two tiles of eight)
# Rows up to which the dispatcher gives a product to the mma.sync kernel; more go the way of 17 and
# more (the gated product to the tcgen05 kernel, the plain ones to the library).  The line was drawn when the kernel cut every product into
# shares (whole decode steps at the 8B shape: 9 rows 4.76 against 4.79 ms, 12 rows 5.30 against 5.24, 16 rows 6.08 against 5.83).  By rows it would
# lie beyond 16: a step at the 1B shape of 12 rows 0.94 ms against 1.17 by the library and the tcgen05 kernel, of 16 rows 0.97 against 1.18; a gated
# MLP of 16 rows, 8B, 59 us against 68; only the 8B attention layer's two products are about 1.5 us faster by the library.
SKINNY_ROWS = 10
MAX_ROWS = 128           # rows the two kernels take between them; beyond this the products are prefill products
# Of 17 to 128 rows the gated product goes to the tcgen05 kernel (47 us against 56 for the library product plus
# gating at the 8B shape and 64 rows).  The plain products do too when TC_PLAIN is set; measured inside a decode
# step the library's are about 7 us a product faster at those sizes, so they stay with the library.
TC_PLAIN = False
SUM_STRIDE = 16          # floats between the sums of squares of two tiles (mma.sync kernel)
_MAX_TILES = 1 << 16
CONSUMER_WARPS = 8       # of a block (GS_CONSUMERS in csrc/gemm_skinny.cu): each may hand over two cut tiles of 16 rows x 16 tokens
_state = {}


def _device_state(device):
    key = device.index
    if key not in _state:
        sms = _library.sm_count()
        counters = torch.zeros(_MAX_TILES, dtype=torch.int32, device=device)
        _library.register_counters(counters)
        partials = torch.empty(max(sms, 1) * CONSUMER_WARPS * 2 * 2 * 128, dtype=torch.float32, device=device)
        _state[key] = (counters, partials, _library.status_word(device))
    return _state[key]


@functools.lru_cache(maxsize=4096)
def _parts(n_out, k, sms):
    """Parts of the sums of squares that a product of these sizes leaves (its plan: of the sizes and ``sms``, the current device's multiprocessors)."""
    return _library.library().dl_gemm_skinny_parts(n_out, k)


def sum_stride(rows):
    """Floats between two parts of the sums of squares that a product of ``rows`` rows leaves."""
    return SUM_STRIDE if rows <= SKINNY_ROWS else gemm_decode_tc.SUM_STRIDE


def takes(x, w, fuse_swiglu=False, max_rows=None):
    M, K = x.shape
    if M > SKINNY_ROWS:
        return (fuse_swiglu or TC_PLAIN) and M <= (max_rows or MAX_ROWS) and gemm_decode_tc.takes(x, w, fuse_swiglu)
    n_out = w.shape[0] // 2 if fuse_swiglu else w.shape[0]
    tiles = (n_out + 7) // 8 if fuse_swiglu else (n_out + 15) // 16
    return (x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16
            and 1 <= M <= min(MAX_ROWS, max_rows or MAX_ROWS)
            and K % 8 == 0 and x.stride(1) == 1 and x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0
            and w.data_ptr() % 16 == 0 and tiles <= _MAX_TILES)


def run(x, w, out_dtype, fuse_swiglu=False, resident=False, row_sums=None, into=None, sizes=None):
    """``row_sums`` = (sums float32 [parts * 16], parts, width, eps): x is a stream times a norm's gain,
    and every output row is multiplied by rsqrt(sum of the row's parts / width + eps); the sums must come
    from a product of the same number of rows (``sum_stride``).
    ``into`` = (stream float32 [M, N], gain float32 [N]): the product is added into the stream in place;
    returns (stream * gain as bfloat16 [M, N], sums of squares float32 [parts * 16]).
    ``sizes``: of x and w, where the caller has them (``product`` in csrc/host/entry.cpp)."""
    M, K, N, x_stride = sizes[:4] if sizes is not None else (*x.shape, w.shape[0], None)
    if M > SKINNY_ROWS:
        return gemm_decode_tc.run(x, w, out_dtype, fuse_swiglu, resident, row_sums, into)
    n_out = N // 2 if fuse_swiglu else N
    counters, partials, status = _device_state(x.device)
    if x_stride is None:
        x_stride = x.stride(0) if M > 1 else max(K, x.stride(0))
    flags = (1 if fuse_swiglu else 0) | (2 if resident else 0)
    tail = (partials, partials.numel(), counters, _MAX_TILES, status, _library.current_stream())
    if row_sums is None and into is None:
        half = out_dtype == torch.bfloat16
        out = _library.empty(M, n_out, out_dtype, x)
        _library.call("dl_gemm_skinny_bf16", x, x_stride, w, out, 1 if half else 0, n_out, M, n_out, K, flags, *tail)
        return out
    sums_in, parts, width, eps = row_sums if row_sums is not None else (None, 0, 1, 0.0)
    if into is not None:
        stream, gain = into
        scaled = _library.empty(M, n_out, torch.bfloat16, x)
        sums_out = torch.empty(_parts(n_out, K, _library.sm_count()) * SUM_STRIDE, dtype=torch.float32, device=x.device)
        out, out_stride, result = stream, stream.stride(0), (scaled, sums_out)
    else:
        gain = scaled = sums_out = None
        out = _library.empty(M, n_out, out_dtype, x)
        out_stride, result = n_out, out
    _library.call("dl_gemm_skinny_fused_bf16", x, x_stride, w, out,
                  0 if out.dtype == torch.float32 else 1, out_stride, M, n_out, K, flags,
                  gain, scaled, n_out,
                  sums_out,
                  sums_in, parts, 1.0 / width, float(eps), *tail)
    return result


def takes_gating(x, w):
    """A gated product with another gating than SwiGLU in its epilogue: the rows of the mma.sync kernel only."""
    return x.shape[0] <= SKINNY_ROWS and takes(x, w, True)


def run_gating(x, w, gate_kind, limit, alpha, resident=False, bias=None):
    """gating(x Wg^T, x Wu^T) in x's dtype for W = [Wg; Wu], the gating ``gate_kind`` of ``ops.GATINGS``, behind ``bias`` (float32
    [2N] or None)."""
    M, K = x.shape
    n_out = w.shape[0] // 2
    counters, partials, status = _device_state(x.device)
    x_stride = x.stride(0) if M > 1 else max(K, x.stride(0))
    out = _library.empty(M, n_out, x.dtype, x)
    _library.call("dl_gemm_skinny_gated_bf16", x, x_stride, w, out, 1, n_out, M, n_out, K,
                  1 | (2 if resident else 0), int(gate_kind), float(limit), float(alpha), bias, partials, partials.numel(),
                  counters, counters.numel(), status, _library.current_stream())
    return out


def run_activated(x, w, kind, resident=False):
    """act(x W^T) in x's dtype for W [N, K] and an activation of one product (``ops.UNGATED``) in the product's epilogue."""
    M, K = x.shape
    n_out = w.shape[0]
    counters, partials, status = _device_state(x.device)
    x_stride = x.stride(0) if M > 1 else max(K, x.stride(0))
    out = _library.empty(M, n_out, x.dtype, x)
    _library.call("dl_gemm_skinny_gated_bf16", x, x_stride, w, out, 1, n_out, M, n_out, K,
                  2 if resident else 0, int(kind), 0.0, 0.0, None, partials, partials.numel(),
                  counters, counters.numel(), status, _library.current_stream())
    return out


def plan(N, K, gated=False, sms=148):
    """How a product is cut on a device of ``sms`` multiprocessors: ("rows", 0, 0, 0), or ("shares", warps of a block with a share, its chunks, blocks)."""
    v = [ctypes.c_int() for _ in range(4)]
    if _library.library().dl_gemm_skinny_plan(N, K, 1 if gated else 0, sms, *(ctypes.byref(i) for i in v)) != 0:
        raise _library.KernelError(f"gemm_skinny: no plan for {N} x {K}")
    return ("rows", 0, 0, 0) if v[0].value else ("shares", v[1].value, v[2].value, v[3].value)


def scratch_need(M, N, K, fuse_swiglu=False, sms=148):
    """(partial floats, counters) the product of these sizes needs."""
    a, b = ctypes.c_int(0), ctypes.c_int(0)
    _library.library().dl_gemm_skinny_scratch(M, N, K, 1 if fuse_swiglu else 0, sms, ctypes.byref(a), ctypes.byref(b))
    return a.value, b.value


def maybe_run(x, w, out_dtype, fuse_swiglu=False, resident=False, sizes=None):
    """y = x W^T (or the gated form) by the skinny kernel when it takes the sizes, else None.
    ``resident``: no work still pending on the stream writes W.  ``sizes`` as in ``run``: they say all that ``takes`` would look up."""
    if sizes is not None and sizes[0] <= SKINNY_ROWS:
        if sizes[4] != 2 or sizes[2] > 16 * _MAX_TILES:
            return None
    elif not takes(x, w, fuse_swiglu):
        return None
    return run(x, w, out_dtype, fuse_swiglu, resident, sizes=sizes)
