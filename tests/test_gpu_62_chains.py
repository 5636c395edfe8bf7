"""The block's one-call inference forward and its gate / up / SiLU autograd function, vs the composition and fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frozen", [(), (0,), (1, 2), (2,)])
@pytest.mark.parametrize("H,I", [(200, 72), (256, 192), (76, 40)])  # narrow rows, the summed kernel, rows of 8-byte multiples
def test_gate_up_silu_backward(cuda, H, I, frozen):
    from qwen3_moe_fused.kernels.fused_mlp import gate_up_silu

    dtype, sizes = torch.bfloat16, [0, 1, 33, 255, 289, 300, 2]
    gen = torch.Generator(device=cuda).manual_seed(3)
    E, M = len(sizes), sum(sizes)
    ts = [(torch.randn(*s, device=cuda, generator=gen) * c).to(dtype) for s, c in
          (((M, H), 1), ((E, I, H), 0.07), ((E, I, H), 0.07))]
    for i, t in enumerate(ts):
        t.requires_grad_(i not in frozen)
    h = gate_up_silu(*ts, torch.tensor(sizes, device=cuda, dtype=torch.int32))
    dh = torch.randn(M, I, device=cuda, generator=gen).to(dtype)
    live = [t for t in ts if t.requires_grad]
    grads = torch.autograd.grad(h, live, dh)
    d = [t.detach().double().requires_grad_(t.requires_grad) for t in ts]
    parts, a = [], 0
    for e, n in enumerate(sizes):
        x = d[0][a:a + n]
        parts.append(torch.nn.functional.silu(x @ d[1][e].T) * (x @ d[2][e].T))
        a += n
    ref = torch.cat(parts)
    # chains of at most six roundings one after the other, each at most 2^-8 of what it applies to: 2-norm over 2-norm
    for got, want in zip((h, *grads), (ref, *torch.autograd.grad(ref, [t for t in d if t.requires_grad], dh.double()))):
        assert (got.double() - want).norm() <= 6 * 2.0 ** -8 * want.norm()
