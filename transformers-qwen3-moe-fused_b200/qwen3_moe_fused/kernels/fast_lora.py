"""Expert MLP with base weights (dense or NF4) plus LoRA on gate / up / down, as one
autograd function with a hand-written backward.

Drop-in for `fast_lora` of the reference (qwen3_moe_fused/kernels/fast_lora.py:66-175):
same 17 positional arguments, gradients for x and the six LoRA matrices only.

    e = G'x   g = U'x   h = silu(e) * g   y = W'h       with  V' = V + s * B A

Differences in how the same quantities are computed:
  * an NF4 base weight is decoded inside the forward GEMM (the reference decodes the
    whole tensor first, :96); the backward decodes it once per projection for dX;
  * LoRA gradients are formed in rank-r space,
        dA = s * (dy B)^T x        dB = s * dy^T (x A^T),
    i.e. two thin grouped GEMMs per matrix, instead of a full (E, out, in) weight-gradient
    GEMM followed by two einsum projections (:139-149);
  * on dense 16-bit weights every `base product + s * (t B)` is one launch that contracts both operand
    pairs into one accumulator (dx: four pairs), with s applied to fp32 accumulators: in bf16 to the thin factor's,
    in fp16 (powers of two) to those of the products with the thin factor, which is held as it is.
"""
import ctypes
import math

import torch

from .. import _lib
from ..grouped_gemm.backward_dw import grouped_gemm_backward_dw
from ..grouped_gemm.forward import grouped_gemm_forward
from ..grouped_gemm.forward_4bit import grouped_gemm_forward_4bit, grouped_gemm_forward_transposed_4bit
from ..grouped_gemm.forward_transposed import grouped_gemm_forward_transposed
from ..grouped_gemm.lora import eligible
from ..quantize.nf4 import dequantize_4bit
from .silu_mul import silu_mul_backward_inplace, silu_mul_forward


def _dense(weight, quant_state, dtype):
    if quant_state is None:
        return weight if weight.dtype == dtype else weight.to(dtype)
    return dequantize_4bit(weight, quant_state, dtype)


def _fits_fused(x, base, quant, adapters, scales, m_sizes) -> bool:
    """Whether the fused form takes the call: dense 16-bit base weights and adapters of matching shapes, ranks that are
    multiples of 8 (16-byte rows of the thin factors; gate and up side by side within the 256 columns of one tile), plain
    numbers as factors.  In fp16 powers of two only, 2^-7..2^7: any other factor would have to go onto the thin factors,
    whose small values it would take low bits from (|s| < 1) or whose large ones it would push out of range (|s| > 1).
    Everything else takes the general form below."""
    if any(q is not None for q in quant) or not all(type(s) in (int, float) and math.isfinite(s) for s in scales):
        return False
    if x.dtype == torch.float16 and not all(math.frexp(abs(s))[0] == 0.5 and 2.0 ** -7 <= abs(s) <= 2.0 ** 7 for s in scales):
        return False
    if not eligible(x, (*base, *adapters), m_sizes):
        return False
    (E, I, H), (Ag, Bg, Au, Bu, Aw, Bw) = base[0].shape, adapters
    if base[1].shape != (E, I, H) or base[2].shape != (E, H, I) or x.shape[1] != H or min(I, H) < 192:
        return False
    rg, ru, rw = Ag.shape[1], Au.shape[1], Aw.shape[1]
    # (the weight gradients of narrow outputs keep six stages and the group tables in shared memory: E <= 192)
    return max(rg, ru, rw) <= 128 and E <= 192 and \
        Ag.shape[2] == H and Au.shape[2] == H and Aw.shape[2] == I and \
        Bg.shape == (E, I, rg) and Bu.shape == (E, I, ru) and Bw.shape == (E, H, rw)


def _still_fits(tensors, shapes, m_sizes) -> bool:
    """Whether what the fused form took or made in the forward can still be read by address: `shapes` as they were, one type
    and device, 16-byte aligned and contiguous, the GEMM path not switched."""
    dtype, device = tensors[0].dtype, tensors[0].get_device()
    for t, shape in zip(tensors, shapes):
        if t.shape != shape or t.dtype != dtype or t.get_device() != device or not t.is_contiguous() or t.data_ptr() % 16:
            return False
    return device >= 0 and m_sizes.get_device() == device and m_sizes.is_contiguous() and m_sizes.numel() == shapes[-1][0] and \
        _lib.load().moe_get_gemm_path() == _lib.PATH_AUTO


def _lora_weights(base, a, b, scales) -> _lib.LoraWeights:
    ptrs = lambda ts: (ctypes.c_void_p * 3)(*(t.data_ptr() for t in ts))
    return _lib.LoraWeights(ptrs(base), ptrs(a), ptrs(b), (ctypes.c_float * 3)(*scales), (ctypes.c_int * 3)(*(t.shape[1] for t in a)))


class FastLora(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, Gq, Gqs, Ag, Bg, Sg, Uq, Uqs, Au, Bu, Su, Wq, Wqs, Aw, Bw, Sw, m_sizes):
        dt = x.dtype
        x = x.contiguous()
        Ag, Bg, Au, Bu, Aw, Bw = (t.to(dt).contiguous() for t in (Ag, Bg, Au, Bu, Aw, Bw))
        if Gqs is None:
            Gq = Gq.to(dt)
        if Uqs is None:
            Uq = Uq.to(dt)
        if Wqs is None:
            Wq = Wq.to(dt)

        ctx.fused = _fits_fused(x, (Gq, Uq, Wq), (Gqs, Uqs, Wqs), (Ag, Bg, Au, Bu, Aw, Bw), (Sg, Su, Sw), m_sizes)
        if ctx.fused:
            M, H, (E, I) = x.shape[0], x.shape[1], Gq.shape[:2]
            # t_gu, t_w: the thin factors of the LoRA products (s x A^T; fp16: +-x A^T), gate and up side by side
            e, g, h, t_gu, t_w, y = (torch.empty((M, n), device=x.device, dtype=dt)
                                     for n in (I, I, I, Ag.shape[1] + Au.shape[1], Aw.shape[1], H))
            w = _lora_weights((Gq, Uq, Wq), (Ag, Au, Aw), (Bg, Bu, Bw), (Sg, Su, Sw))
            ms = _lib.as_index_tensor(m_sizes)
            with torch.cuda.device(x.device):
                status = _lib.load().moe_lora_mlp_fwd(
                    ctypes.addressof(w), x.data_ptr(), ms.data_ptr(), _lib.int_code(ms.dtype), e.data_ptr(), g.data_ptr(),
                    h.data_ptr(), t_gu.data_ptr(), t_w.data_ptr(), y.data_ptr(), M, H, I, E, _lib.float_code(dt),
                    _lib.stream_ptr(x.device))
            _lib.check(status, "moe_lora_mlp_fwd")
            ctx.custom_saved_tensors = (Gq, Gqs, Sg, Uq, Uqs, Su, Wq, Wqs, Sw, m_sizes)
            saved = (x, Ag, Bg, Au, Bu, Aw, Bw, e, g, t_gu, t_w)
            ctx.save_for_backward(*saved)
            ctx.shapes = [t.shape for t in (*saved, Gq, Uq, Wq)]
            return y

        def base(_x, _wq, _wqs):
            if _wqs is None:
                return grouped_gemm_forward(_x, _wq, m_sizes, dt)
            return grouped_gemm_forward_4bit(_x, _wq, _wqs, m_sizes, dt)

        def mv_lora(_x, _wq, _wqs, _a, _b, _s):
            _y = base(_x, _wq, _wqs)
            _y += grouped_gemm_forward(grouped_gemm_forward(_x, _a, m_sizes, dt), _b, m_sizes, dt) * _s
            return _y

        e = mv_lora(x, Gq, Gqs, Ag, Bg, Sg)
        g = mv_lora(x, Uq, Uqs, Au, Bu, Su)
        h = silu_mul_forward(e, g)
        y = mv_lora(h, Wq, Wqs, Aw, Bw, Sw)

        ctx.custom_saved_tensors = (Gq, Gqs, Sg, Uq, Uqs, Su, Wq, Wqs, Sw, m_sizes)
        ctx.save_for_backward(x, Ag, Bg, Au, Bu, Aw, Bw, e, g)
        return y

    @staticmethod
    def backward(ctx, dy):
        Gq, Gqs, Sg, Uq, Uqs, Su, Wq, Wqs, Sw, m_sizes = ctx.custom_saved_tensors
        saved = ctx.saved_tensors
        x, Ag, Bg, Au, Bu, Aw, Bw, e, g = saved[:9]
        # (since the forward the GEMM path may have been switched, base weights moved, saved tensors changed by hooks: the
        # fused form takes addresses, the general form's launchers check each operand)
        if ctx.fused and _still_fits((*saved, Gq, Uq, Wq), ctx.shapes, m_sizes):
            return FastLora._backward_fused(ctx, dy, saved)
        dt = x.dtype
        dy = dy.contiguous().to(dt)

        def vm(_x, _w):  # rows times (E, k, n) weight read transposed
            return grouped_gemm_forward_transposed(_x, _w, m_sizes, dt)

        def vm_base(_x, _wq, _wqs):  # the same through a base weight that may be NF4 (decoded inside the kernel)
            if _wqs is None:
                return vm(_x, _wq)
            return grouped_gemm_forward_transposed_4bit(_x, _wq, _wqs, m_sizes, dt)

        def mv(_x, _w):
            return grouped_gemm_forward(_x, _w, m_sizes, dt)

        def vv(_y, _x):  # per-expert _y^T _x
            return grouped_gemm_backward_dw(_x, _y, m_sizes, dt)

        # down projection
        dyB = vm(dy, Bw)  # (rows, r)
        dh = vm_base(dy, Wq, Wqs)
        dh += vm(dyB, Aw) * Sw
        # dh, e, g become h, de, dg
        silu_mul_backward_inplace(dh, e, g)
        h, de, dg = dh, e, g
        del dh, e, g

        dAw = vv(dyB, h) * Sw
        dBw = vv(dy, mv(h, Aw)) * Sw

        dgB = vm(dg, Bu)
        dAu = vv(dgB, x) * Su
        dBu = vv(dg, mv(x, Au)) * Su

        deB = vm(de, Bg)
        dAg = vv(deB, x) * Sg
        dBg = vv(de, mv(x, Ag)) * Sg

        dx = None
        if ctx.needs_input_grad[0]:
            dx = vm_base(de, Gq, Gqs)
            dx += vm(deB, Ag) * Sg
            dx += vm_base(dg, Uq, Uqs)
            dx += vm(dgB, Au) * Su

        return (dx, None, None, dAg, dBg, None, None, None, dAu, dBu, None, None, None, dAw, dBw, None, None)


    @staticmethod
    def _backward_fused(ctx, dy, saved):
        Gq, _, Sg, Uq, _, Su, Wq, _, Sw, m_sizes = ctx.custom_saved_tensors
        x, Ag, Bg, Au, Bu, Aw, Bw, e, g, t_gu, t_w = saved
        dy = dy.contiguous().to(x.dtype)
        if dy.data_ptr() % 16:
            dy = dy.clone()
        M, H, (E, I) = x.shape[0], x.shape[1], Gq.shape[:2]
        code = _lib.float_code(x.dtype)
        dAg, dAu, dAw, dBg, dBu, dBw, d_gu, d_w = (torch.empty_like(t) for t in (Ag, Au, Aw, Bg, Bu, Bw, t_gu, t_w))
        dh = torch.empty_like(e)
        dx = torch.empty_like(x) if ctx.needs_input_grad[0] else None
        w = _lora_weights((Gq, Uq, Wq), (Ag, Au, Aw), (Bg, Bu, Bw), (Sg, Su, Sw))
        grads = _lib.LoraGrads((ctypes.c_void_p * 3)(dAg.data_ptr(), dAu.data_ptr(), dAw.data_ptr()),
                               (ctypes.c_void_p * 3)(dBg.data_ptr(), dBu.data_ptr(), dBw.data_ptr()))
        ms = _lib.as_index_tensor(m_sizes)
        lib = _lib.load()
        ws_ptr, ws_bytes = _lib.workspace(x.device, lib.moe_grouped_gemm_workspace_bytes(2, M, H, I, E))
        with torch.cuda.device(x.device):
            status = lib.moe_lora_mlp_bwd(  # overwrites dh, e, g with h, de, dg
                ctypes.addressof(w), ctypes.addressof(grads), dy.data_ptr(), x.data_ptr(), ms.data_ptr(), _lib.int_code(ms.dtype),
                e.data_ptr(), g.data_ptr(), t_gu.data_ptr(), t_w.data_ptr(), dh.data_ptr(), d_gu.data_ptr(), d_w.data_ptr(),
                _lib.ptr(dx), M, H, I, E, code, ws_ptr, ws_bytes, _lib.stream_ptr(x.device))
        _lib.check(status, "moe_lora_mlp_bwd")
        return (dx, None, None, dAg, dBg, None, None, None, dAu, dBu, None, None, None, dAw, dBw, None, None)


fast_lora = FastLora.apply
