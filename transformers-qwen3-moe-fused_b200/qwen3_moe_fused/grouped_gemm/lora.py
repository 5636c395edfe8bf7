"""Launchers of the grouped GEMMs whose operands are sums or slices: several (activation, weight) pairs into one
result, thin LoRA projections with a factor, and weight gradients of column slices.

No counterpart in the reference, which adds and scales the products of separate launches
(qwen3_moe_fused/kernels/fast_lora.py:101-153).
"""
import ctypes
from typing import Optional

import torch

from .. import _lib


def eligible(x: torch.Tensor, weights, m_sizes: torch.Tensor) -> bool:
    """True if the tensor-core kernels take these operands: x (M, K) and 3-D weights, 16-bit, 16-byte aligned, every
    extent a multiple of 8, and no other kernel family selected."""
    if not (x.is_cuda and x.ndim == 2 and x.dtype in (torch.bfloat16, torch.float16) and x.is_contiguous() and x.shape[0] > 0):
        return False
    if not (m_sizes.device == x.device and m_sizes.ndim == 1 and _lib.is_int_tensor(m_sizes) and m_sizes.is_contiguous()):
        return False
    E = m_sizes.numel()
    if not 1 <= E <= 1024 or x.data_ptr() % 16 or x.shape[1] % 8 or _lib.load().moe_get_gemm_path() != _lib.PATH_AUTO:
        return False
    for w in weights:
        if w.device != x.device or w.dtype != x.dtype or w.ndim != 3 or w.shape[0] != E or not w.is_contiguous():
            return False
        if w.data_ptr() % 16 or w.shape[1] % 8 or w.shape[2] % 8 or w.numel() == 0:
            return False
    return True


def grouped_gemm_sum(pairs, m_sizes: torch.Tensor, transposed: bool) -> Optional[torch.Tensor]:
    """sum_i x_i W_i^T (W_i (E, N, K_i)), or with `transposed` sum_i x_i W_i (W_i (E, K_i, N)); x_i (M, K_i) may be a
    column slice.  One accumulator, one rounding.  None if the kernel does not cover the operands."""
    x0, w0 = pairs[0]
    M, N, E = x0.shape[0], w0.shape[2 if transposed else 1], w0.shape[0]
    n = len(pairs)
    y = torch.empty((M, N), device=x0.device, dtype=x0.dtype)
    xs = (ctypes.c_void_p * n)(*(x.data_ptr() for x, _ in pairs))
    ws = (ctypes.c_void_p * n)(*(w.data_ptr() for _, w in pairs))
    lds = (ctypes.c_int64 * n)(*(x.stride(0) for x, _ in pairs))
    ks = (ctypes.c_int * n)(*(x.shape[1] for x, _ in pairs))
    m_sizes = _lib.as_index_tensor(m_sizes)
    with torch.cuda.device(x0.device):
        status = _lib.load().moe_grouped_gemm_sum(
            int(transposed), n, xs, lds, ws, ks, _lib.ptr(m_sizes), _lib.int_code(m_sizes.dtype), _lib.ptr(y), M, N, E,
            _lib.float_code(x0.dtype), _lib.stream_ptr(x0.device))
    if status == _lib.ERR_UNSUPPORTED:
        return None
    _lib.check(status, "moe_grouped_gemm_sum")
    return y


def lora_project(x: torch.Tensor, a0: torch.Tensor, s0: float, m_sizes: torch.Tensor, out: torch.Tensor,
                 a1: Optional[torch.Tensor] = None, s1: float = 1.0, transposed: bool = False) -> None:
    """out[:, :n0] = s0 * x a0^T, out[:, n0:] = s1 * x a1^T with a_i (E, n_i, K); `transposed`: out = s0 * x a0 with a0
    (E, K, n0).  `out` may be a column slice.  The factor multiplies the fp32 accumulator."""
    n0 = a0.shape[2 if transposed else 1]
    m_sizes = _lib.as_index_tensor(m_sizes)
    with torch.cuda.device(x.device):
        status = _lib.load().moe_lora_project(
            int(transposed), _lib.ptr(x), _lib.ptr(a0), n0, float(s0), _lib.ptr(a1),
            0 if a1 is None else a1.shape[1], float(s1), _lib.ptr(m_sizes), _lib.int_code(m_sizes.dtype), _lib.ptr(out),
            out.stride(0), x.shape[0], x.shape[1], a0.shape[0], _lib.float_code(x.dtype), _lib.stream_ptr(x.device))
    _lib.check(status, "moe_lora_project")


def grouped_gemm_dw_strided(x: torch.Tensor, dy: torch.Tensor, m_sizes: torch.Tensor, n1: int = 0):
    """`grouped_gemm_backward_dw` on operands that may be column slices: w[e] = sum over the rows of e of dy^T x.  With
    `n1` the columns of dy belong to two weights: (E, n1, K) and (E, N - n1, K) are returned."""
    M, K = x.shape
    N, E = dy.shape[1], m_sizes.numel()
    w = torch.empty((E, n1 or N, K), device=x.device, dtype=x.dtype)
    w2 = torch.empty((E, N - n1, K), device=x.device, dtype=x.dtype) if n1 else None
    lib = _lib.load()
    m_sizes = _lib.as_index_tensor(m_sizes)
    ws_ptr, ws_bytes = _lib.workspace(x.device, lib.moe_grouped_gemm_workspace_bytes(2, M, N, K, E))
    with torch.cuda.device(x.device):
        status = lib.moe_grouped_gemm_dw_strided(
            _lib.ptr(x), x.stride(0), _lib.ptr(dy), dy.stride(0), _lib.ptr(m_sizes), _lib.int_code(m_sizes.dtype), _lib.ptr(w),
            _lib.ptr(w2), n1, M, N, K, E, _lib.float_code(x.dtype), ws_ptr, ws_bytes, _lib.stream_ptr(x.device))
    _lib.check(status, "moe_grouped_gemm_dw_strided")
    return (w, w2) if n1 else w
