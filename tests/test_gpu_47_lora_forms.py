"""The two forms of fast_lora on dense weights, one accumulator per projection and the general composition: which calls take
which, and what each gives, vs the same MLP in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROUND = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}  # relative error of one rounding, at most


def case(dev, dtype=torch.bfloat16, ranks=(16, 16, 16), scales=(2.0, 2.0, 2.0), sizes=(0, 5, 100, 33, 64), H=256, I=192,
         a_scale=(1.0, 1.0, 1.0), b_scale=0.1, frozen_x=False, seed=0):
    """Arguments of fast_lora (without m_sizes), m_sizes, the tensors it differentiates."""
    gen = torch.Generator(device=dev).manual_seed(seed)
    E, M = len(sizes), sum(sizes)

    def normal(*shape, s):
        return (torch.randn(*shape, device=dev, generator=gen) * s).to(dtype)

    x = normal(M, H, s=1).requires_grad_(not frozen_x)
    args, leaves = [x], [x]
    for (n_out, n_in), r, s, c in zip(((I, H), (I, H), (H, I)), ranks, scales, a_scale):
        a, b = normal(E, r, n_in, s=c * n_in ** -0.5), normal(E, n_out, r, s=b_scale)
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


class Number(float):
    """A factor that only the general form takes."""


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("scales,a_scale,b_scale,dy_scale", [
    ((1 / 16, 1 / 16, 1 / 16), (1, 1, 1), 0.01, 2e-3),   # thin factors whose low bits a factor below 1 would take (fp16)
    ((-1 / 128, 128.0, 1 / 128), (1, 1e-2, 1), 0.01, 0.1),  # both ends of the range, and both signs
    ((2.0, 16.0, 2.0), (1e4, 3e3, 1), 2e-4, 1e-3),        # thin factors that a factor above 1 would push out of range (fp16)
])
def test_factors_cost_no_precision(cuda, dtype, scales, a_scale, b_scale, dy_scale):
    """One accumulator per projection is no further from fp64 than the general form, whatever the factors do."""
    from qwen3_moe_fused.kernels.fast_lora import fast_lora

    err = []
    for fused in (True, False):
        args, m_sizes, leaves = case(cuda, dtype, scales=scales, a_scale=a_scale, b_scale=b_scale)
        call = args if fused else [Number(a) if isinstance(a, float) else a for a in args]
        y = fast_lora(*call, m_sizes)
        assert y.grad_fn.fused == fused
        dy = (torch.randn(y.shape, device=cuda, generator=torch.Generator(device=cuda).manual_seed(9)) * dy_scale).to(dtype)
        err.append(errors((y, *torch.autograd.grad(y, leaves, dy)), reference(args, m_sizes, leaves, dy)))
    # fewer roundings one after the other in the fused form; 5 % for the chance in sums of differently rounded terms
    for got, general in zip(*err):
        assert got <= 1.05 * general, err


@pytest.mark.parametrize("fused,change", [
    (True, {}),
    (True, {"frozen_x": True}),
    (True, {"ranks": (128, 64, 128)}), (False, {"ranks": (136, 8, 8)}), (False, {"ranks": (8, 8, 12)}),
    (True, {"I": 200, "H": 192}), (False, {"I": 184}), (False, {"H": 184}),
    (True, {"sizes": [1] * 191 + [40]}), (False, {"sizes": [1] * 192 + [40]}),
    (True, {"dtype": torch.float16, "scales": (0.5, 1.0, -4.0)}), (False, {"dtype": torch.float16, "scales": (0.5, 1.5, 1.0)}),
    (True, {"dtype": torch.float16, "scales": (128.0, 1.0, 2.0 ** -7)}), (False, {"dtype": torch.float16, "scales": (256.0, 1.0, 1.0)}),
    (False, {"dtype": torch.float16, "scales": (1.0, 2.0 ** -8, 1.0)}), (False, {"dtype": torch.float16, "scales": (1.0, 0.0, 1.0)}),
    (True, {"scales": (0.7, 0.0, 300.0)}),
])
def test_which_form(cuda, fused, change):
    """Both sides of every limit of the rule, and the result on each."""
    from qwen3_moe_fused import _lib
    from qwen3_moe_fused.kernels.fast_lora import fast_lora

    dtype = change.get("dtype", torch.bfloat16)
    args, m_sizes, leaves = case(cuda, b_scale=0.02, **change)
    y = fast_lora(*args, m_sizes)
    assert y.grad_fn.fused == fused
    dy = torch.randn_like(y)
    wanted = [t for t in leaves if t.requires_grad]
    grads = torch.autograd.grad(y, wanted, dy)
    ref = reference(args, m_sizes, leaves, dy)
    if len(wanted) < len(leaves):
        ref = (ref[0], *ref[2:])
    for g, r in zip((y, *grads), ref):
        # chains of at most six roundings one after the other, each at most ROUND of what it applies to
        assert (g.double() - r).norm() <= 6 * ROUND[dtype] * r.norm()
    assert _lib.read_error_flag() == 0


@pytest.mark.parametrize("which", ["hook", "moved base"])
def test_backward_checks_what_it_reads(cuda, which):
    """The backward in one accumulator per projection takes addresses: saved tensors that hooks gave back with other strides,
    and base weights that left the device since the forward, are refused as in the general form."""
    from qwen3_moe_fused.kernels.fast_lora import fast_lora

    args, m_sizes, leaves = case(cuda)
    if which == "hook":
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t.mT.contiguous().mT):
            y = fast_lora(*args, m_sizes)
    else:
        y = fast_lora(*args, m_sizes)
        args[11].data = args[11].data.cpu()
    assert y.grad_fn.fused
    with pytest.raises(AssertionError):
        torch.autograd.grad(y, leaves, torch.ones_like(y))


def test_backward_with_saved_tensors_on_the_host(cuda):
    """Saved on the host and brought back unchanged: the same bits."""
    from qwen3_moe_fused.kernels.fast_lora import fast_lora

    args, m_sizes, leaves = case(cuda)
    dy = torch.randn_like(args[0])
    want = torch.autograd.grad(fast_lora(*args, m_sizes), leaves, dy)
    with torch.autograd.graph.save_on_cpu():
        y = fast_lora(*args, m_sizes)
    assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(y, leaves, dy), want))
