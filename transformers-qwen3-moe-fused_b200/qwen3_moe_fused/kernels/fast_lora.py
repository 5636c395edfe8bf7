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
    pairs into one accumulator (dx: four pairs), with s applied to the fp32 accumulator of the thin factor.
"""
import math

import torch

from ..grouped_gemm.backward_dw import grouped_gemm_backward_dw
from ..grouped_gemm.forward import grouped_gemm_forward
from ..grouped_gemm.forward_4bit import grouped_gemm_forward_4bit, grouped_gemm_forward_transposed_4bit
from ..grouped_gemm.forward_transposed import grouped_gemm_forward_transposed
from ..grouped_gemm.lora import eligible, grouped_gemm_dw_strided, grouped_gemm_sum, lora_project
from ..quantize.nf4 import dequantize_4bit
from .silu_mul import silu_mul_backward_inplace, silu_mul_forward


def _dense(weight, quant_state, dtype):
    if quant_state is None:
        return weight if weight.dtype == dtype else weight.to(dtype)
    return dequantize_4bit(weight, quant_state, dtype)


def _fits_fused(x, base, quant, adapters, scales, m_sizes) -> bool:
    """Whether the fused form takes the call: dense 16-bit base weights and adapters of matching shapes, ranks that are
    multiples of 8 (16-byte rows of the thin factors; gate and up side by side within the 256 columns of one tile), plain
    numbers as factors.  In fp16 the factor moves onto the thin product, so it must not be able to push that out of
    range: 1/16..16 is four of the format's 30 binades.  Everything else takes the general form below."""
    if any(q is not None for q in quant) or not all(type(s) in (int, float) and math.isfinite(s) for s in scales):
        return False
    if x.dtype == torch.float16 and not all(1 / 16 <= abs(s) <= 16 for s in scales):
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
            M, rg, rw = x.shape[0], Ag.shape[1], Aw.shape[1]
            # thin factors of the LoRA products, already scaled: gate and up side by side (x is read once), down
            t_gu = torch.empty((M, rg + Au.shape[1]), device=x.device, dtype=dt)
            lora_project(x, Ag, Sg, m_sizes, t_gu, Au, Su)
            e = grouped_gemm_sum(((x, Gq), (t_gu[:, :rg], Bg)), m_sizes, False)
            g = grouped_gemm_sum(((x, Uq), (t_gu[:, rg:], Bu)), m_sizes, False)
            h = silu_mul_forward(e, g)
            t_w = torch.empty((M, rw), device=x.device, dtype=dt)
            lora_project(h, Aw, Sw, m_sizes, t_w)
            y = grouped_gemm_sum(((h, Wq), (t_w, Bw)), m_sizes, False)
            ctx.custom_saved_tensors = (Gq, Gqs, Sg, Uq, Uqs, Su, Wq, Wqs, Sw, m_sizes)
            ctx.save_for_backward(x, Ag, Bg, Au, Bu, Aw, Bw, e, g, t_gu, t_w)
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
        if ctx.fused:
            return FastLora._backward_fused(ctx, dy)
        Gq, Gqs, Sg, Uq, Uqs, Su, Wq, Wqs, Sw, m_sizes = ctx.custom_saved_tensors
        x, Ag, Bg, Au, Bu, Aw, Bw, e, g = ctx.saved_tensors
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
    def _backward_fused(ctx, dy):
        Gq, _, Sg, Uq, _, Su, Wq, _, Sw, m_sizes = ctx.custom_saved_tensors
        x, Ag, Bg, Au, Bu, Aw, Bw, e, g, t_gu, t_w = ctx.saved_tensors
        rg = Ag.shape[1]
        dy = dy.contiguous().to(x.dtype)
        if dy.data_ptr() % 16:
            dy = dy.clone()

        d_w = torch.empty_like(t_w)  # s dy B
        lora_project(dy, Bw, Sw, m_sizes, d_w, transposed=True)
        dh = grouped_gemm_sum(((dy, Wq), (d_w, Aw)), m_sizes, True)
        # dh, e, g become h, de, dg
        silu_mul_backward_inplace(dh, e, g)
        h, de, dg = dh, e, g
        del dh, e, g
        dAw = grouped_gemm_dw_strided(h, d_w, m_sizes)
        dBw = grouped_gemm_dw_strided(t_w, dy, m_sizes)
        d_gu = torch.empty_like(t_gu)  # [s de B | s dg B]
        lora_project(de, Bg, Sg, m_sizes, d_gu[:, :rg], transposed=True)
        lora_project(dg, Bu, Su, m_sizes, d_gu[:, rg:], transposed=True)
        dAg = grouped_gemm_dw_strided(x, d_gu[:, :rg], m_sizes)
        dAu = grouped_gemm_dw_strided(x, d_gu[:, rg:], m_sizes)
        dBg = grouped_gemm_dw_strided(t_gu[:, :rg], de, m_sizes)
        dBu = grouped_gemm_dw_strided(t_gu[:, rg:], dg, m_sizes)
        dx = None
        if ctx.needs_input_grad[0]:
            dx = grouped_gemm_sum(((de, Gq), (d_gu[:, :rg], Ag), (dg, Uq), (d_gu[:, rg:], Au)), m_sizes, True)
        return (dx, None, None, dAg, dBg, None, None, None, dAu, dBu, None, None, None, dAw, dBw, None, None)


fast_lora = FastLora.apply
