"""Grouped GEMMs over several operand pairs, thin projections and strided weight gradients, and the form of fast_lora
that uses them, vs the same sums in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROUND = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}  # relative error of one rounding, at most
SIZES = [0, 1, 16, 17, 33, 255, 0, 256, 257, 288, 289, 300, 544, 2]  # edges of the 256-token tiles, their tails, 32-row rounds


def groups(m_sizes):
    a = 0
    for e, n in enumerate(m_sizes):
        yield e, slice(a, a + n)
        a += n


def check(got, ref, mag, terms, dtype):
    """|got - ref| within one rounding of the result plus the fp32 accumulation of `terms` products of total size `mag`."""
    bound = 1.01 * ROUND[dtype] * ref.abs() + terms * 2.0 ** -23 * mag + 2.0 ** -24
    assert ((got.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("N,ks", [(192, (64, 8)), (264, (72, 16)), (256, (8,)), (512, (200, 24, 136, 40)), (776, (128, 64))])
def test_sum_of_pairs(cuda, dtype, transposed, N, ks):
    from qwen3_moe_fused import _lib
    from qwen3_moe_fused.grouped_gemm.lora import grouped_gemm_sum

    gen = torch.Generator(device=cuda).manual_seed(N)
    E, M = len(SIZES), sum(SIZES)
    m_sizes = torch.tensor(SIZES, device=cuda, dtype=torch.int32)
    wide = torch.randn(M, sum(ks), device=cuda, generator=gen).to(dtype)
    xs = list(wide.split(ks, 1))  # column slices of one tensor
    ws = [torch.randn((E, k, N) if transposed else (E, N, k), device=cuda, generator=gen).to(dtype) for k in ks]
    y = grouped_gemm_sum(list(zip(xs, ws)), m_sizes, transposed)
    ref = torch.zeros(M, N, device=cuda, dtype=torch.float64)
    mag = torch.zeros_like(ref)
    for x, w in zip(xs, ws):
        for e, r in groups(SIZES):
            we = w[e].double() if transposed else w[e].double().T
            ref[r] += x[r].double() @ we
            mag[r] += x[r].double().abs() @ we.abs()
    check(y, ref, mag, sum(ks), dtype)
    assert _lib.read_error_flag() == 0


@pytest.mark.parametrize("K", [64, 200])
@pytest.mark.parametrize("n0,n1", [(8, 0), (16, 16), (24, 8), (64, 64), (128, 128), (40, 0)])
def test_projections_and_strided_dw(cuda, K, n0, n1):
    from qwen3_moe_fused.grouped_gemm.lora import grouped_gemm_dw_strided, lora_project

    dtype = torch.bfloat16
    gen = torch.Generator(device=cuda).manual_seed(n0 + K)
    E, M = len(SIZES), sum(SIZES)
    m_sizes = torch.tensor(SIZES, device=cuda, dtype=torch.int64)
    x = torch.randn(M, K, device=cuda, generator=gen).to(dtype)
    a0, a1 = (torch.randn(E, max(n, 8), K, device=cuda, generator=gen).to(dtype) for n in (n0, n1))
    out = torch.full((M, n0 + n1 + 8), 7.0, device=cuda, dtype=dtype)  # eight columns to the right stay as they are
    lora_project(x, a0, 1.75, m_sizes, out, a1 if n1 else None, -0.375)
    back = torch.full((M, n0 + 8), 7.0, device=cuda, dtype=dtype)
    lora_project(x, a0.transpose(1, 2).contiguous(), 1.75, m_sizes, back[:, :n0], transposed=True)
    dw = grouped_gemm_dw_strided(x, out[:, :n0], m_sizes)
    dwt = grouped_gemm_dw_strided(out[:, :n0], x, m_sizes)
    both = None
    if 0 < n1 and n0 + n1 <= 128:  # two weights that share x
        both = torch.cat(grouped_gemm_dw_strided(x, out[:, :n0 + n1], m_sizes, n1=n0), 1)
    for e, r in groups(SIZES):
        xd = x[r].double()
        for cols, a, s in ((slice(0, n0), a0, 1.75), (slice(n0, n0 + n1), a1, -0.375)):
            if cols.start == cols.stop:
                continue
            ref, mag = s * (xd @ a[e].double().T), abs(s) * (xd.abs() @ a[e].double().T.abs())
            check(out[r, cols], ref, mag, K + 2, dtype)
            if cols.start == 0:
                check(back[r, :n0], ref, mag, K + 2, dtype)
        t = out[r, :n0].double()
        check(dw[e], t.T @ xd, t.abs().T @ xd.abs(), r.stop - r.start + 2, dtype)
        if both is not None:
            tb = out[r, :n0 + n1].double()
            check(both[e], tb.T @ xd, tb.abs().T @ xd.abs(), r.stop - r.start + 2, dtype)
        check(dwt[e], xd.T @ t, xd.abs().T @ t.abs(), r.stop - r.start + 2, dtype)
    assert (out[:, n0 + n1:] == 7.0).all() and (back[:, n0:] == 7.0).all()


@pytest.mark.parametrize("dtype,ranks,scales", [(torch.bfloat16, (16, 16, 16), (2.0, 2.0, 2.0)),
                                                (torch.float16, (8, 24, 64), (0.7, 1.5, -3.0)),
                                                (torch.bfloat16, (128, 64, 128), (0.25, 0.5, 1.0)),
                                                (torch.bfloat16, (4, 4, 4), (2.0, 2.0, 2.0))])  # the last: the general form
def test_fast_lora_forms(cuda, dtype, ranks, scales):
    from qwen3_moe_fused.kernels.fast_lora import fast_lora

    gen = torch.Generator(device=cuda).manual_seed(sum(ranks))
    sizes = [0, 5, 300, 33, 64]
    E, M, H, I = len(sizes), sum(sizes), 256, 192
    m_sizes = torch.tensor(sizes, device=cuda, dtype=torch.int32)

    def normal(*shape, s):
        return (torch.randn(*shape, device=cuda, generator=gen) * s).to(dtype)

    def mlp(x, ws):
        outs = []
        for e, r in groups(sizes):
            def proj(t, w, a, b, s):
                return t @ w[e].T + s * (t @ a[e].T) @ b[e].T
            outs.append(proj(torch.nn.functional.silu(proj(x[r], *ws[0])) * proj(x[r], *ws[1]), *ws[2]))
        return torch.cat(outs)

    x = normal(M, H, s=1).requires_grad_()
    args, leaves, base = [x], [x], []
    for (n_out, n_in), r, s in zip(((I, H), (I, H), (H, I)), ranks, scales):
        w, a, b = normal(E, n_out, n_in, s=0.06), normal(E, r, n_in, s=n_in ** -0.5), normal(E, n_out, r, s=0.1)
        args += [w, None, a.requires_grad_(), b.requires_grad_(), s]
        leaves += [a, b]
        base.append(w)
    y = fast_lora(*args, m_sizes)
    dy = normal(M, H, s=1)
    grads = torch.autograd.grad(y, leaves, dy)
    d = [t.detach().double().requires_grad_() for t in leaves]
    ref = mlp(d[0], [(base[i].double(), d[1 + 2 * i], d[2 + 2 * i], scales[i]) for i in range(3)])
    rgrads = torch.autograd.grad(ref, d, dy.double())
    # chains of at most six roundings one after the other (the products of the general form are rounded apart from their
    # sums), each at most ROUND of what it applies to: 2-norm over 2-norm
    for got, want in zip((y, *grads), (ref, *rgrads)):
        assert (got.double() - want).norm() <= 6 * ROUND[dtype] * want.norm()
