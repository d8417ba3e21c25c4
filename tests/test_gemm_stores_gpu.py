"""Results of the dense and grouped products inside larger buffers: nothing beside them is written, whichever way they leave."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(*shape):
    return torch.randn(*shape, device="cuda").bfloat16()


def _room(rows, cols, first):
    """A result of `cols` columns from column `first` on of a wider buffer with more rows, all 7."""
    wide = torch.full((rows + 40, first + cols + 72 - (first + cols) % 8), 7.0, device="cuda", dtype=torch.bfloat16)
    return wide, wide[:rows, first:first + cols]


def _check(wide, got, ref, rows=None):
    """Products of unit normals: fp32 sums and one rounding to bf16 (2^-9, doubled); `rows`: those that are written (None: all)."""
    seen = torch.ones(got.shape[0], dtype=torch.bool, device="cuda") if rows is None else rows
    assert ((got.double() - ref).abs()[seen] <= 2.0 ** -8 * ref.abs()[seen] + 1e-3).all()
    keep = torch.ones_like(wide, dtype=torch.bool)
    first = (got.data_ptr() - wide.data_ptr()) // 2
    keep[:got.shape[0], first:first + got.shape[1]] = ~seen.unsqueeze(1)
    assert (wide[keep] == 7.0).all()


# tiles of every width, the paired kernel (512) and the rule's own choice (0); rows around 32 and 128, columns around 64; results that
# TMA can address (column 8) and that it cannot (column 3)
@pytest.mark.parametrize("bn", [0, 64, 128, 256, 512])
@pytest.mark.parametrize("M,N", [(1, 8), (31, 64), (33, 72), (40, 72), (127, 129), (261, 328), (264, 200),
                                 (513, 520), (520, 328)])
@pytest.mark.parametrize("first", [8, 3])
def test_dense_results_stay_in_their_place(bn, M, N, first):
    from trainscale_b200.ops import _lib, gemm
    torch.manual_seed(0)
    K = 136
    a, b = _rand(M, K), _rand(N, K)
    ref = a.double() @ b.double().t()
    wide, out = _room(M, N, first)
    gemm.matmul_nt(a, b, out=out, bn=bn)
    _check(wide, out, ref)
    if M % 8 == 0 and N % 8 == 0:                       # operands that are read across their rows
        wide, out = _room(M, N, first)
        gemm.matmul_nn(a, b.t().contiguous(), out=out, bn=bn)
        _check(wide, out, ref)
        wide, out = _room(M, N, first)
        gemm.matmul_tn(a.t().contiguous(), b.t().contiguous(), out=out, bn=bn)
        _check(wide, out, ref)
    torch.cuda.synchronize()
    _lib.raise_on_any_device_error()


# both sides of the lines: 256 x 256 tiles for every pair of SMs; 128 x 128 tiles for every SM; fewer than either
@pytest.mark.parametrize("M,N", [(1000, 4096), (500, 3072), (1024, 2304), (1024, 2432), (2048, 2048), (300, 8192), (256, 19072)])
def test_the_rules_choice_gives_the_bits_of_every_tile(M, N):
    from trainscale_b200.ops import gemm
    torch.manual_seed(0)
    a, b = _rand(M, 192), _rand(N, 192)
    ref = a.double() @ b.double().t()
    wide, out = _room(M, N, 8)
    gemm.matmul_nt(a, b, out=out)
    _check(wide, out, ref)
    for bn in (128, 512):
        assert torch.equal(gemm.matmul_nt(a, b, bn=bn), out), bn


@pytest.mark.parametrize("N", [64, 136, 200, 328])
@pytest.mark.parametrize("first", [8, 3])
def test_grouped_rows_stay_in_their_place(N, first):
    """Tiles of three experts, one of them without rows, and tiles of none, which are left alone."""
    from trainscale_b200.ops import moe
    torch.manual_seed(0)
    E, K = 3, 64
    experts = torch.tensor([0, 0, 2, -1, 2], dtype=torch.int32, device="cuda")
    P = 128 * len(experts)
    a, w = _rand(P, K), _rand(E, N, K)
    wide, out = _room(P, N, first)
    moe._grouped(1, a, w, out, P, N, K, K, K, out.stride(0), False, False, False, experts, E)
    e = experts.long().repeat_interleave(128)
    ref = torch.einsum("pk,pnk->pn", a.double(), w.double()[e.clamp(min=0)])
    _check(wide, out, ref, e >= 0)


@pytest.mark.parametrize("M", [128, 256, 96])          # whole tiles leave by TMA, partial ones would reach into the next slab
@pytest.mark.parametrize("N", [64, 200, 328])
@pytest.mark.parametrize("first", [8, 3])
def test_grouped_reductions_stay_in_their_slabs(M, N, first):
    """Three slabs, the one in the middle of an expert without rows: zeros."""
    from trainscale_b200.ops import moe
    torch.manual_seed(0)
    seg = torch.tensor([0, 256, 256, 384], dtype=torch.int32, device="cuda")
    a, b = _rand(384, M), _rand(384, N)
    wide, out = _room(3 * M, N, first)
    moe._grouped(2, a, b, out, M, N, 384, M, N, out.stride(0), True, True, False, seg, 3)
    at = seg.tolist()
    ref = torch.cat([a[s:t].double().t() @ b[s:t].double() for s, t in zip(at, at[1:])])
    _check(wide, out, ref)
    assert (out[M:2 * M] == 0).all()
