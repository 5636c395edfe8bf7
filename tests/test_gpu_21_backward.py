"""Backward kernels of the routing path vs autograd of the same operations in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROUND = {torch.float32: 2.0 ** -23, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}  # relative error of one rounding, at most


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("T,k,H", [(1, 1, 8), (3, 8, 2048), (37, 4, 1000), (5, 8, 2056), (7, 3, 37), (2500, 8, 64)])
def test_combine_backward(cuda, dtype, T, k, H):
    from qwen3_moe_fused.kernels.routing import combine

    gen = torch.Generator().manual_seed(T * 1000 + H)
    inv = torch.randperm(T * k, generator=gen)
    sort = torch.argsort(inv)
    y, w, dout = (torch.randn(*s, generator=gen).to(dtype) for s in ((T * k, H), (T, k), (T, H)))
    yd, wd = y.double().requires_grad_(), w.double().requires_grad_()
    ref = torch.einsum("tkh,tk->th", yd[inv].view(T, k, H), wd)
    rdy, rdw = torch.autograd.grad(ref, (yd, wd), dout.double())
    ii, si = inv.to(torch.int32).to(cuda), sort.to(torch.int32).to(cuda)
    for need_y, need_w in ((True, True), (True, False), (False, True)):
        yc, wc = y.to(cuda).requires_grad_(need_y), w.to(cuda).requires_grad_(need_w)
        leaves = [t for t in (yc, wc) if t.requires_grad]
        grads = list(torch.autograd.grad(combine(yc, si, ii, wc), leaves, dout.to(cuda)))
        if need_y:  # one product, rounded once (fp16 results below 2^-14 have a fixed spacing of 2^-24)
            assert ((grads.pop(0).cpu().double() - rdy).abs() <= 1.01 * ROUND[dtype] * rdy.abs() + 2.0 ** -24).all()
        if need_w:  # fp32 sum of H products in some order, then one rounding
            bound = (dout.double().unsqueeze(1) * y.double()[inv].view(T, k, H)).abs().sum(-1) * (H + 2) * 2.0 ** -24
            assert ((grads.pop(0).cpu().double() - rdw).abs() <= bound + 1.01 * ROUND[dtype] * rdw.abs() + 2.0 ** -24).all()


@pytest.mark.parametrize("norm", [True, False])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,E,k", [(1, 128, 8), (61, 128, 8), (9, 5, 2), (33, 200, 20), (4, 1024, 32), (3000, 32, 4)])
def test_router_backward(cuda, T, E, k, dtype, norm):
    from qwen3_moe_fused.kernels.routing import softmax_topk_autograd

    gen = torch.Generator().manual_seed(E + T)
    logits, dw = torch.randn(T, E, generator=gen).to(dtype), torch.randn(T, k, generator=gen).to(dtype)
    lg = logits.to(cuda).requires_grad_()
    weights, experts = softmax_topk_autograd(lg, k, norm, dtype)
    (grad,) = torch.autograd.grad(weights, lg, dw.to(cuda))
    ld = logits.double().requires_grad_()
    p = torch.softmax(ld, 1)
    sel = p.gather(1, experts.cpu())
    out = sel / sel.sum(-1, keepdim=True) if norm else sel
    (ref,) = torch.autograd.grad(out, ld, dw.double())
    # fp32 arithmetic: each of the k terms behind an element is of the size p * max|dw| (over the winners' sum when they
    # are renormalised) and carries some ten roundings of exp, sums over E and k, and quotients
    scale = dw.double().abs().amax(1, keepdim=True) * p.detach()
    if norm:
        scale = scale / sel.detach().sum(-1, keepdim=True)
    bound = 64 * 2.0 ** -24 * k * scale + 1.01 * ROUND[dtype] * ref.abs() + 1e-30
    assert ((grad.cpu().double() - ref).abs() <= bound).all()


def test_combine_backward_twice(cuda):
    """Gradients taken with create_graph can be differentiated again, in y, the weights and dout."""
    from qwen3_moe_fused.kernels.routing import combine

    T, k, H = 5, 2, 24
    gen = torch.Generator().manual_seed(0)
    inv = torch.randperm(T * k, generator=gen)
    ii, si = inv.to(torch.int32).to(cuda), torch.argsort(inv).to(torch.int32).to(cuda)
    ts = [torch.randn(*s, generator=gen) for s in ((T * k, H), (T, k), (T, H))]
    g = [t.to(cuda).requires_grad_() for t in ts]
    d = [t.double().requires_grad_() for t in ts]

    def twice(out, y, w, dout):
        dy, dw = torch.autograd.grad(out, (y, w), dout, create_graph=True)
        return torch.autograd.grad(dy.square().sum() + dw.square().sum(), (y, w, dout))

    got = twice(combine(g[0], si, ii, g[1]), *g)
    ref = twice(torch.einsum("tkh,tk->th", d[0][inv].view(T, k, H), d[1]), *d)
    for a, b in zip(got, ref):  # fp32 sums of up to H * k products of products
        assert (a.cpu().double() - b).norm() <= 1e-5 * b.norm()


@pytest.mark.parametrize("norm", [False, True])
def test_batched_gradients(cuda, norm):
    """Several gradients at once through the router, and through the combine where only its weights want one: each as if it
    had come alone."""
    from qwen3_moe_fused.kernels.routing import combine, softmax_topk_autograd

    T, E, k, H = 5, 12, 3, 24
    gen = torch.Generator(device=cuda).manual_seed(0)
    logits = torch.randn(T, E, device=cuda, generator=gen).requires_grad_()
    weights, _ = softmax_topk_autograd(logits, k, norm, torch.float32)
    inv = torch.randperm(T * k, device=cuda, generator=gen)
    y = torch.randn(T * k, H, device=cuda, generator=gen)
    w = weights.detach().requires_grad_()
    out = combine(y, torch.argsort(inv).to(torch.int32), inv.to(torch.int32), w)
    v_weights = torch.randn(4, T, k, device=cuda, generator=gen)
    v_out = torch.randn(4, T, H, device=cuda, generator=gen)

    def pull(res, leaf):
        return lambda v: torch.autograd.grad(res, leaf, v, retain_graph=True)[0]

    got = [torch.autograd.grad(weights, logits, v_weights, is_grads_batched=True, retain_graph=True)[0],
           torch.func.vmap(pull(out, w))(v_out)]
    want = [torch.stack([pull(res, leaf)(v) for v in vs]) for res, leaf, vs in ((weights, logits, v_weights), (out, w, v_out))]
    for a, b in zip(got, want):  # fp32 sums in another order
        assert (a - b).norm() <= 1e-5 * b.norm()


def test_hooks_that_change_layout_or_type(cuda):
    """What saved-tensor hooks give back with other strides or in another type still gives the gradients it holds."""
    from qwen3_moe_fused.kernels.routing import combine, softmax_topk_autograd

    T, E, k, H = 5, 12, 3, 24
    gen = torch.Generator(device=cuda).manual_seed(0)
    logits = torch.randn(T, E, device=cuda, generator=gen).requires_grad_()
    inv = torch.randperm(T * k, device=cuda, generator=gen)
    sort_idx, inv = torch.argsort(inv).to(torch.int32), inv.to(torch.int32)
    y = torch.randn(T * k, H, device=cuda, generator=gen).to(torch.bfloat16).requires_grad_()
    dout = torch.randn(T, H, device=cuda, generator=gen).to(torch.bfloat16)

    def grads():
        weights, _ = softmax_topk_autograd(logits, k, True, torch.bfloat16)
        return torch.autograd.grad(combine(y, sort_idx, inv, weights), (y, logits), dout)

    def other_strides(t):
        return t.mT.contiguous().mT if t.ndim == 2 else t

    def other_type(t):
        return t.float() if t.dtype == torch.bfloat16 else t

    want = grads()
    for change in (other_strides, other_type):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, change):
            got = grads()
        for a, b in zip(got, want):  # one rounding to bf16 on either side
            assert (a.double() - b.double()).norm() <= 2.0 ** -7 * b.double().norm()
