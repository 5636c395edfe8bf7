"""The two forms of fast_lora on dense weights, one accumulator per projection and the general composition: which calls take
which, and what each gives, vs the same MLP in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROUND = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}  # relative error of one rounding, at most


def case(dev, dtype=torch.bfloat16, ranks=(16, 16, 16), scales=(2.0, 2.0, 2.0), sizes=(0, 5, 100, 33, 64), H=256, I=192,
         a_scale=1.0, b_scale=0.1, frozen_x=False, seed=0):
    """Arguments of fast_lora (without m_sizes), m_sizes, the tensors it differentiates."""
    gen = torch.Generator(device=dev).manual_seed(seed)
    E, M = len(sizes), sum(sizes)

    def normal(*shape, s):
        return (torch.randn(*shape, device=dev, generator=gen) * s).to(dtype)

    x = normal(M, H, s=1).requires_grad_(not frozen_x)
    args, leaves = [x], [x]
    for (n_out, n_in), r, s in zip(((I, H), (I, H), (H, I)), ranks, scales):
        a, b = normal(E, r, n_in, s=a_scale * n_in ** -0.5), normal(E, n_out, r, s=b_scale)
        args += [normal(E, n_out, n_in, s=0.06), None, a.requires_grad_(), b.requires_grad_(), s]
        leaves += [a, b]
    return args, torch.tensor(sizes, device=dev, dtype=torch.int32), leaves


def reference(args, m_sizes, leaves, dy):
    """y and the gradients of `leaves` in fp64."""
    d = [t.detach().double().requires_grad_() for t in leaves]
    outs, a = [], 0
    for e, n in enumerate(m_sizes.tolist()):
        def proj(t, i):
            return t @ args[1 + 5 * i][e].double().T + args[5 + 5 * i] * (t @ d[1 + 2 * i][e].T) @ d[2 + 2 * i][e].T
        x = d[0][a:a + n]
        outs.append(proj(torch.nn.functional.silu(proj(x, 0)) * proj(x, 1), 2))
        a += n
    y = torch.cat(outs)
    return (y, *torch.autograd.grad(y, d, dy.double()))


def errors(got, ref):
    return [((g.double() - r).norm() / r.norm()).item() for g, r in zip(got, ref)]


def test_backward_after_the_path_was_switched(cuda):
    """What a forward in one accumulator saved is enough for the general backward."""
    from qwen3_moe_fused import _lib
    from qwen3_moe_fused.kernels.fast_lora import fast_lora

    args, m_sizes, leaves = case(cuda)
    y = fast_lora(*args, m_sizes)
    assert y.grad_fn.fused
    dy = torch.randn_like(y)
    _lib.set_gemm_path(_lib.PATH_SIMT)
    try:
        grads = torch.autograd.grad(y, leaves, dy)
    finally:
        _lib.set_gemm_path(_lib.PATH_AUTO)
    # chains of at most six roundings one after the other, each at most ROUND of what it applies to
    assert max(errors((y, *grads), reference(args, m_sizes, leaves, dy))) <= 6 * ROUND[torch.bfloat16]
