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


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,E,k,H,I,norm", [(1, 128, 8, 256, 64, True), (3, 8, 8, 200, 72, False), (257, 5, 2, 64, 200, True),
                                            (300, 128, 8, 520, 192, True)])
def test_block_call_equals_composition(cuda, dtype, T, E, k, H, I, norm):
    """Same kernels in the same order, so the same bits."""
    from qwen3_moe_fused.functional import moe_fused_linear
    from qwen3_moe_fused.kernels.fused_mlp import gate_up_silu_forward
    from qwen3_moe_fused.kernels.indexing import get_expert_counts_and_idx
    from qwen3_moe_fused.kernels.routing import combine, gather_rows
    from qwen3_moe_fused.moe_block import _block_infer, moe_block_forward, route

    gen = torch.Generator(device=cuda).manual_seed(T)
    x, gw, gp, up, dp = ((torch.randn(*s, device=cuda, generator=gen) * 0.1).to(dtype)
                         for s in ((T, H), (E, H), (E, I, H), (E, I, H), (E, H, I)))
    with torch.no_grad():
        logits = torch.nn.functional.linear(x, gw)
        w, sel = route(logits, k, norm, dtype)
        m_sizes, si, ii = get_expert_counts_and_idx(sel.view(T * k), E)
        y = moe_fused_linear(gate_up_silu_forward(gather_rows(x, si, ii, k), gp, up, m_sizes), dp, m_sizes)
        want = combine(y, si, ii, w)
        assert torch.equal(_block_infer(x, logits, gp, up, dp, k, norm), want)
        out, lg = moe_block_forward(x.view(1, T, H), gw, gp, up, dp, k, norm)
        assert torch.equal(out.view(T, H), want) and torch.equal(lg, logits)
        # an up projection that is not 16-byte aligned takes the composition
        odd = torch.empty(up.numel() + 1, device=cuda, dtype=dtype)[1:].view_as(up).copy_(up)
        assert _block_infer(x, logits, gp, odd, dp, k, norm) is None
        out, _ = moe_block_forward(x.view(1, T, H), gw, gp, odd, dp, k, norm)
        assert torch.allclose(out.view(T, H).float(), want.float(), rtol=2e-2, atol=2e-3 * want.float().abs().max().item())


@pytest.mark.parametrize("which", range(5))  # tokens, router, gate, up, down
def test_block_refuses_forward_mode(cuda, which):
    """No kernel here carries a forward-mode derivative, and `no_grad` does not switch that mode off: a tangent is refused,
    not dropped."""
    import torch.autograd.forward_ad as fw
    from qwen3_moe_fused.moe_block import moe_block_forward

    T, E, k, H, I = 3, 8, 2, 256, 64
    ts = [torch.ones(s, device=cuda, dtype=torch.bfloat16) for s in ((1, T, H), (E, H), (E, I, H), (E, I, H), (E, H, I))]
    with torch.no_grad(), fw.dual_level():
        moe_block_forward(*ts, k)  # inside a level, but without a tangent
        ts[which] = fw.make_dual(ts[which], torch.ones_like(ts[which]))
        with pytest.raises(NotImplementedError):
            moe_block_forward(*ts, k)
