"""Dispatch to the float32 product on the tensor cores (csrc/gemm_f32_tc.cu)."""
from __future__ import annotations

import ctypes
import functools

import torch

from . import library as _library

_P, _I, _L = _library._P, _library._I, ctypes.c_longlong
_library.register_signatures({
    "dl_gemm_f32_tc": [_P, _I, _P, _P, _I, _I, _I, _I, _P, _L, _P, _L, _I, _P, _P],
    "dl_gemm_f32_tc_scratch": [_I, _I, _I, _I, _P, _P],
})

# The rule looks at the matrix alone, never at the rows: both products give the same bits for any number of rows, but not the
# same bits as each other, and a model's steps of any size must agree.  Measured (a kernel from a captured graph, 1 / 16 / 64 /
# 1,000 rows, this product against FFMA, us): K 256, N 16: 3.9 / 4.1 / 7.0 / 8.2 against 5.3 / 5.4 / 15 / 32; K 256, N 2,048: 4.5 /
# 5.8 / 9.9 / 19 against 5.6 / 5.6 / 17 / 43; K 2,048, N 2,048: 8.5 / 9.9 / 15 / 59 against 35 / 36 / 125 / 267; but K 128, N 2,048:
# 4.9 / 4.9 / 6.7 / 12 against 3.4 / 3.5 / 9.1 / 27.  Below 16 outputs a tile of 128 would be empty.
MIN_K, MIN_N = 256, 16
SELF_SPLIT = 32          # FT_SELF_SPLIT in csrc/gemm_f32_tc.cu: so few rows are read by the copy engine as they are (16-byte aligned)


def takes(w):
    """Is y = x W^T for this float32 W [N, K] the tensor cores' for any number of rows?"""
    N, K = w.shape
    return K >= MIN_K and N >= MIN_N and K % 4 == 0 and w.data_ptr() % 16 == 0


@functools.lru_cache(maxsize=4096)
def scratch_need(M, N, K, sms):
    """(bfloat16 values of planes, floats of sums) the product of these sizes needs."""
    planes, sums = _L(0), _L(0)
    _library.library().dl_gemm_f32_tc_scratch(M, N, K, sms, ctypes.byref(planes), ctypes.byref(sums))
    return planes.value, sums.value


def run(x, x_stride, w, resident=False):
    """y = x W^T, float32 [M, N]; x [M, K] with rows ``x_stride`` apart."""
    M, K = x.shape
    N = w.shape[0]
    y = _library.empty(M, N, torch.float32, x)
    if M == 0:
        return y
    if M <= SELF_SPLIT and (x_stride % 4 or x.data_ptr() % 16):
        x, x_stride = _library.empty(M, K, torch.float32, x).copy_(x), K
    n_planes, n_sums = scratch_need(M, N, K, _library.sm_count())
    scratch = torch.empty(n_sums + (n_planes + 1) // 2, dtype=torch.float32, device=x.device) if n_sums or n_planes else None
    at = 0 if scratch is None else scratch.data_ptr()      # the planes (a multiple of 8 values a row) in front, the sums behind
    _library.call("dl_gemm_f32_tc", x, x_stride, w, y, N, M, N, K, at, n_planes, at + 2 * n_planes, n_sums,
                  1 if resident else 0, _library.status_word(x.device).data_ptr(), _library.current_stream())
    return y
