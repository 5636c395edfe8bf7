"""What lies next to a group of rows: every length of a group's last reduction block, and infinities and NaN in the rows on
either side of a group and behind the last one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def restore_path():
    from qwen3_moe_fused import _lib

    yield
    _lib.set_gemm_path(_lib.PATH_AUTO)
    assert _lib.read_error_flag() == 0


def groups(sizes):
    a = 0
    for e, n in enumerate(sizes):
        yield e, slice(a, a + n)
        a += n


@pytest.mark.parametrize("repeat,N,K,path", [  # CTA pairs; one CTA with 256 (four and, from 222 experts on, three stages) and 128 columns
    (1, 200, 264, "AUTO"), (1, 136, 256, "TC_SINGLE"), (4, 136, 256, "TC_SINGLE"), (1, 136, 96, "TC_SINGLE")])
@pytest.mark.parametrize("last", [1, 7, 16, 61])  # the group that ends with the tensor
def test_dw_every_residue(cuda, repeat, N, K, path, last):
    """Groups of 0..64 rows: every number of rows in a group's last 64 and in its last 16."""
    from qwen3_moe_fused import _lib
    from qwen3_moe_fused.grouped_gemm.backward_dw import grouped_gemm_backward_dw

    _lib.set_gemm_path(getattr(_lib, "PATH_" + path))
    gen = torch.Generator(device=cuda).manual_seed(N + last)
    sizes = [n for _ in range(repeat) for n in range(65)] + [last]
    M = sum(sizes)
    x, dy = (torch.randn(M, n, device=cuda, generator=gen).to(torch.bfloat16) for n in (K, N))
    dw = grouped_gemm_backward_dw(x, dy, torch.tensor(sizes, device=cuda, dtype=torch.int32), torch.bfloat16).double()
    for e, r in groups(sizes):
        xd, dd = x[r].double(), dy[r].double()
        ref, mag = dd.T @ xd, dd.abs().T @ xd.abs()
        # one rounding to bf16, and the fp32 accumulation of the products
        assert ((dw[e] - ref).abs() <= 1.01 * 2.0 ** -8 * ref.abs() + (r.stop - r.start + 2) * 2.0 ** -23 * mag).all(), sizes[e]


@pytest.mark.parametrize("path", ["AUTO", "TC_SINGLE"])
@pytest.mark.parametrize("poisoned", [0, 1])  # the groups with infinities and NaN: every second one
def test_infinities_stay_in_their_group(cuda, path, poisoned):
    """The other groups' results are the same bits as without them."""
    from qwen3_moe_fused import _lib
    from qwen3_moe_fused.grouped_gemm.backward_dw import grouped_gemm_backward_dw
    from qwen3_moe_fused.grouped_gemm.forward import grouped_gemm_forward
    from qwen3_moe_fused.grouped_gemm.forward_transposed import grouped_gemm_forward_transposed
    from qwen3_moe_fused.grouped_gemm.lora import grouped_gemm_dw_strided, grouped_gemm_sum, lora_project
    from qwen3_moe_fused.kernels.fused_mlp import gate_up_silu_forward

    _lib.set_gemm_path(getattr(_lib, "PATH_" + path))
    gen = torch.Generator(device=cuda).manual_seed(1)
    sizes = list(range(1, 35)) + [0, 64, 65, 111, 257, 300]
    sizes = [sizes[i] for i in torch.randperm(len(sizes), generator=torch.Generator().manual_seed(2)).tolist()]
    E, rows, behind = len(sizes), sum(sizes), 40  # rows behind the last group belong to nobody
    H, I, r = 256, 200, 16
    m_sizes = torch.tensor(sizes, device=cuda, dtype=torch.int32)

    def normal(*shape):
        return torch.randn(*shape, device=cuda, generator=gen).to(torch.bfloat16)

    x, dy, thin, gate, up, a = normal(rows + behind, H), normal(rows + behind, I), normal(rows + behind, 2 * r), normal(E, I, H), \
        normal(E, I, H), normal(E, r, H)
    clean = [e for e in range(E) if e % 2 != poisoned]
    bad = torch.ones(rows + behind, device=cuda, dtype=torch.bool)
    for e, s in groups(sizes):
        if e in clean:
            bad[s] = False
    kinds = torch.tensor([float("inf"), float("-inf"), float("nan")], device=cuda, dtype=torch.bfloat16)

    def results(x, dy, thin):
        out = {"fwd": grouped_gemm_forward(x, gate, m_sizes), "dx": grouped_gemm_forward_transposed(dy, gate, m_sizes),
               "thin fwd": grouped_gemm_forward(x, a, m_sizes), "dw": grouped_gemm_backward_dw(x, dy, m_sizes, torch.bfloat16),
               "thin dw": grouped_gemm_backward_dw(thin, dy, m_sizes, torch.bfloat16),
               "fp32 dw": grouped_gemm_backward_dw(x, dy, m_sizes, torch.float32),
               "two dw": torch.cat(grouped_gemm_dw_strided(x, thin, m_sizes, n1=r), 1),
               "project": torch.empty(rows + behind, 2 * r, device=cuda, dtype=torch.bfloat16)}
        lora_project(x, a, 0.5, m_sizes, out["project"], a, 2.0)
        if path == "AUTO":
            out["sum"] = grouped_gemm_sum(((dy, gate), (dy, up), (thin[:, r:], a)), m_sizes, True)
            out["gate up"] = gate_up_silu_forward(x, gate, up, m_sizes)
        return out

    def poison(t):
        cols = torch.arange(t.shape[1], device=cuda)
        return torch.where(bad[:, None], kinds[(torch.arange(t.shape[0], device=cuda)[:, None] + cols) % 3], t)

    want, got = results(x, dy, thin), results(poison(x), poison(dy), poison(thin))
    for name, ref in want.items():
        if ref.ndim == 3:
            assert torch.equal(got[name][clean], ref[clean]), name
        else:
            assert torch.equal(got[name][~bad], ref[~bad]), name
            assert not torch.isnan(ref[~bad].float()).any(), name
