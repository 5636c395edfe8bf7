"""Router and token movement kernels of the sparse MoE block.

These replace sequences of ATen calls inside the reference block forward
(qwen3_moe_fused/modular_qwen3_moe_fused.py:87-115): softmax -> topk -> renormalise ->
cast; expand -> gather; un-permute -> weighted sum.
"""
import torch

from .. import _lib


def _is_batched(t: torch.Tensor) -> bool:
    """Whether `t` stands for several gradients at once (torch.func.vmap, or is_grads_batched of torch.autograd.grad).  Such a
    tensor has no address for a kernel; ATen operations take it."""
    return torch._C._functorch.is_batchedtensor(t) or torch._C._functorch.is_legacy_batchedtensor(t)


def _addressable(like: torch.Tensor, *tensors: torch.Tensor) -> bool:
    """Whether a kernel may read these next to `like`: saved-tensor hooks may have given back another device or layout."""
    return all(t.device == like.device and t.is_contiguous() for t in tensors)


@torch.no_grad()
def softmax_topk(router_logits: torch.Tensor, k: int, norm_topk_prob: bool, out_dtype: torch.dtype):
    """(weights (T,k) out_dtype, experts (T,k) int64); winners ordered by probability
    descending, equal probabilities by ascending expert id."""
    assert router_logits.is_cuda and router_logits.ndim == 2 and router_logits.is_contiguous()
    T, E = router_logits.shape
    weights = torch.empty((T, k), device=router_logits.device, dtype=out_dtype)
    experts = torch.empty((T, k), device=router_logits.device, dtype=torch.int64)
    with torch.cuda.device(router_logits.device):
        status = _lib.load().moe_router_softmax_topk(
            _lib.ptr(router_logits), _lib.float_code(router_logits.dtype), T, E, k, int(norm_topk_prob),
            _lib.ptr(weights), _lib.float_code(out_dtype), _lib.ptr(experts), _lib.stream_ptr(router_logits.device),
        )
    _lib.check(status, "moe_router_softmax_topk")
    return weights, experts


class SoftmaxTopk(torch.autograd.Function):
    """Differentiable wrapper: the forward is one kernel; the backward is one kernel that
    recomputes the fp32 softmax of the (T, E) logits and differentiates gather -> renormalise
    -> cast, which is what autograd does for the reference's sequence of ATen calls."""

    @staticmethod
    def forward(ctx, router_logits, k, norm_topk_prob, out_dtype):
        weights, experts = softmax_topk(router_logits, k, norm_topk_prob, out_dtype)
        ctx.save_for_backward(router_logits, experts)
        ctx.norm = norm_topk_prob
        ctx.mark_non_differentiable(experts)
        return weights, experts

    @staticmethod
    def backward(ctx, dweights, _dexperts):
        logits, experts = ctx.saved_tensors
        if _is_batched(dweights) or not _addressable(dweights, logits, experts) or experts.dtype != torch.int64:
            with torch.enable_grad():
                lg = logits.detach().requires_grad_()
                sel = torch.softmax(lg, dim=1, dtype=torch.float32).gather(1, experts)
                if ctx.norm:
                    sel = sel / sel.sum(dim=-1, keepdim=True)
                (grad,) = torch.autograd.grad(sel.to(dweights.dtype), lg, dweights)
            return grad, None, None, None
        T, E = logits.shape
        dweights = dweights.contiguous()
        grad = torch.empty_like(logits)
        with torch.cuda.device(logits.device):
            status = _lib.load().moe_router_softmax_topk_bwd(
                _lib.ptr(logits), _lib.float_code(logits.dtype), _lib.ptr(experts), _lib.ptr(dweights),
                _lib.float_code(dweights.dtype), T, E, experts.shape[1], int(ctx.norm), _lib.ptr(grad),
                _lib.stream_ptr(logits.device),
            )
        _lib.check(status, "moe_router_softmax_topk_bwd")
        return grad, None, None, None


def softmax_topk_autograd(router_logits, k, norm_topk_prob, out_dtype):
    return SoftmaxTopk.apply(router_logits, k, norm_topk_prob, out_dtype)


def _gather_rows(hidden: torch.Tensor, sort_idx: torch.Tensor, k: int) -> torch.Tensor:
    assert hidden.is_cuda and hidden.ndim == 2 and hidden.is_contiguous()
    assert sort_idx.dtype == torch.int32 and sort_idx.is_contiguous()
    rows = sort_idx.numel()
    out = torch.empty((rows, hidden.shape[1]), device=hidden.device, dtype=hidden.dtype)
    with torch.cuda.device(hidden.device):
        status = _lib.load().moe_gather_rows(
            _lib.ptr(hidden), _lib.ptr(sort_idx), k, _lib.ptr(out), rows, hidden.shape[1],
            _lib.float_code(hidden.dtype), _lib.stream_ptr(hidden.device),
        )
    _lib.check(status, "moe_gather_rows")
    return out


def _expand_rows(hidden: torch.Tensor, inv_sort_idx: torch.Tensor, k: int) -> torch.Tensor:
    """The result of _gather_rows computed through the inverse index (out[inv_sort_idx[t*k+j]] =
    hidden[t]): every token row is read once instead of k times."""
    assert hidden.is_cuda and hidden.ndim == 2 and hidden.is_contiguous()
    assert inv_sort_idx.dtype == torch.int32 and inv_sort_idx.is_contiguous()
    tokens = hidden.shape[0]
    assert inv_sort_idx.numel() == tokens * k
    out = torch.empty((tokens * k, hidden.shape[1]), device=hidden.device, dtype=hidden.dtype)
    with torch.cuda.device(hidden.device):
        status = _lib.load().moe_expand_rows(
            _lib.ptr(hidden), _lib.ptr(inv_sort_idx), k, _lib.ptr(out), tokens, hidden.shape[1],
            _lib.float_code(hidden.dtype), _lib.stream_ptr(hidden.device),
        )
    _lib.check(status, "moe_expand_rows")
    return out


def _combine(y: torch.Tensor, inv_sort_idx: torch.Tensor, weights: torch.Tensor) -> torch.Tensor:
    assert y.is_cuda and y.ndim == 2 and y.is_contiguous()
    assert inv_sort_idx.dtype == torch.int32 and inv_sort_idx.is_contiguous()
    assert weights.is_contiguous() and weights.dtype == y.dtype
    T, k = weights.shape
    out = torch.empty((T, y.shape[1]), device=y.device, dtype=y.dtype)
    with torch.cuda.device(y.device):
        status = _lib.load().moe_combine(
            _lib.ptr(y), _lib.ptr(inv_sort_idx), _lib.ptr(weights), _lib.ptr(out), T, k, y.shape[1],
            _lib.float_code(y.dtype), _lib.stream_ptr(y.device),
        )
    _lib.check(status, "moe_combine")
    return out


class GatherRows(torch.autograd.Function):
    """out[j] = hidden[sort_idx[j] // k].  Backward: each token sums the gradients of its k copies."""

    @staticmethod
    def forward(ctx, hidden, sort_idx, inv_sort_idx, k):
        ctx.save_for_backward(inv_sort_idx)
        ctx.k = k
        if inv_sort_idx.numel() == hidden.shape[0] * k:
            return _expand_rows(hidden, inv_sort_idx, k)  # same rows, each token read once
        return _gather_rows(hidden, sort_idx, k)

    @staticmethod
    def backward(ctx, dout):
        (inv_sort_idx,) = ctx.saved_tensors
        k = ctx.k
        T = inv_sort_idx.numel() // k
        ones = torch.ones((T, k), device=dout.device, dtype=dout.dtype)
        return _combine(dout.contiguous(), inv_sort_idx, ones), None, None, None


class Combine(torch.autograd.Function):
    """out[t] = sum_j weights[t, j] * y[inv_sort_idx[t*k + j]]."""

    @staticmethod
    def forward(ctx, y, sort_idx, inv_sort_idx, weights):
        ctx.save_for_backward(y, sort_idx, inv_sort_idx, weights)
        return _combine(y, inv_sort_idx, weights)

    @staticmethod
    def backward(ctx, dout):
        y, sort_idx, inv_sort_idx, weights = ctx.saved_tensors
        T, k = weights.shape
        dout = dout.contiguous()
        dy = dw = None
        # create_graph wants operations that autograd can follow a second time
        if torch.is_grad_enabled() or _is_batched(dout) or not _addressable(dout, y, sort_idx, inv_sort_idx, weights) or \
                not y.dtype == weights.dtype == dout.dtype or inv_sort_idx.dtype != torch.int32:
            if ctx.needs_input_grad[0]:
                dy = gather_rows(dout, sort_idx, inv_sort_idx, k) * weights.reshape(-1)[sort_idx.long()].unsqueeze(1)
            if ctx.needs_input_grad[3]:
                dw = torch.einsum("tkh,th->tk", y[inv_sort_idx.long()].view(T, k, -1).float(), dout.float()).to(weights.dtype)
            return dy, None, None, dw
        if ctx.needs_input_grad[0]:
            dy = torch.empty((T * k, y.shape[1]), device=y.device, dtype=y.dtype)
        if ctx.needs_input_grad[3]:
            dw = torch.empty((T, k), device=y.device, dtype=weights.dtype)
        with torch.cuda.device(y.device):
            status = _lib.load().moe_combine_bwd(
                _lib.ptr(dout), _lib.ptr(y), _lib.ptr(inv_sort_idx), _lib.ptr(weights), _lib.ptr(dy), _lib.ptr(dw),
                T, k, y.shape[1], _lib.float_code(y.dtype), _lib.stream_ptr(y.device),
            )
        _lib.check(status, "moe_combine_bwd")
        return dy, None, None, dw


def gather_rows(hidden, sort_idx, inv_sort_idx, k):
    return GatherRows.apply(hidden, sort_idx, inv_sort_idx, k)


def combine(y, sort_idx, inv_sort_idx, weights):
    return Combine.apply(y, sort_idx, inv_sort_idx, weights)
