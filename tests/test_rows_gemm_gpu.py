"""Products of up to 256 rows by weight tiles (csrc/rows_gemm.cu) against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# rows: MMA widths (multiples of 16) and their neighbours, whole and partial second blocks of 128
ROWS = [1, 2, 15, 16, 17, 33, 64, 97, 128, 129, 256]


def _run(x, w, cols, dtype, glu=-1):
    """The kernel whatever the rule of the dispatch says."""
    from trainscale_b200.ops import gemm
    return gemm._stream_rows(x, w, cols, dtype, glu)


def _exact(x, w):
    return x.double() @ w.double().t()


# columns: whole and partial 128-wide tiles, not a multiple of four; reductions: less than a block, a partial block, every split
@pytest.mark.parametrize("N,K", [(128, 64), (130, 8), (129, 200), (2048, 2048), (384, 8192), (64, 1032), (40000, 256)])
@pytest.mark.parametrize("fp32", [False, True])
def test_products_match_fp64(N, K, fp32):
    from trainscale_b200.ops import _lib
    torch.manual_seed(0)
    w = torch.randn(N, K, device="cuda").bfloat16()
    for M in ROWS:
        x = torch.randn(M, K + 8, device="cuda").bfloat16()[:, :K]           # rows with a stride of their own
        y, again = (_run(x, w, N, torch.float32 if fp32 else x.dtype) for _ in range(2))
        ref = _exact(x, w)
        torch.cuda.synchronize()
        _lib.raise_on_any_device_error()
        # fp32 sums of K products (each rounding at most 2^-23 of the sum of magnitudes so far), then one rounding to bf16
        bound = 2.0 ** -23 * K * (x.double().abs() @ w.double().abs().t()) + (0 if fp32 else 2.0 ** -8) * ref.abs() + 1e-6
        assert ((y.double() - ref).abs() <= bound).all(), (M, float((y.double() - ref).abs().max()))
        assert torch.equal(y, again), M


@pytest.mark.parametrize("act", ["silu", "gelu", "gelu_tanh"])
@pytest.mark.parametrize("I,K", [(64, 64), (72, 200), (1000, 512), (8192, 2048)])
def test_gated_products_match_fp64(I, K, act):
    from trainscale_b200.ops import _lib, activation
    torch.manual_seed(0)
    w = (torch.randn(2 * I, K, device="cuda") / K ** 0.5).bfloat16()
    for M in ROWS:
        x = torch.randn(M, K, device="cuda").bfloat16()
        y = _run(x, w, I, x.dtype, activation._ACT[act])
        torch.cuda.synchronize()
        _lib.raise_on_any_device_error()
        g, u = _exact(x, w).chunk(2, -1)
        a = torch.nn.functional.silu(g) if act == "silu" else \
            torch.nn.functional.gelu(g, approximate="tanh" if act == "gelu_tanh" else "none")
        # one rounding to bf16 and fp32 sums of unit size, whose error the other factor scales
        assert ((y.double() - a * u).abs() <= 2.0 ** -8 * (a * u).abs() + 2.0 ** -17 * (1 + g.abs()) * (1 + u.abs())).all(), M


@pytest.mark.parametrize("M,N,K", [(64, 12352, 64), (65, 12352, 64), (128, 256, 64), (129, 256, 64), (256, 64, 192), (257, 64, 192),
                                   (3, 100, 60)])
def test_every_route_of_the_dispatch(M, N, K):
    """Both sides of each line of the rule, and rows that are no 16-byte vectors."""
    from trainscale_b200.ops import gemm
    torch.manual_seed(0)
    w, x = torch.randn(N, K, device="cuda").bfloat16(), torch.randn(M, K, device="cuda").bfloat16()
    if K % 8:
        assert not gemm._streamed(x, w)
        return
    ref = _exact(x, w)
    for dtype in (None, torch.float32):
        assert ((gemm.step_linear(x, w, dtype).double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-3).all()
    half = ref[:, :N // 2]
    y = gemm.step_glu(x, w, "silu").double() - torch.nn.functional.silu(half) * ref[:, N // 2:]
    # two roundings of gate and up to bf16 where the product is not fused
    assert (y.abs() <= 2.0 ** -6 * (1 + half.abs()) * (1 + ref[:, N // 2:].abs())).all()


@pytest.mark.parametrize("N,K", [(128, 64), (2048, 2048), (384, 8192), (64, 16384)])
def test_fp32_results_and_partial_sums_keep_fp32(N, K):
    """Relative to the norm of the result: K products added in fp32, a bit of 2^-24 lost at random (or, as tensor cores add, always
    towards zero: 2^-24 for each of the K / 16 steps) stays below 1e-5 * max(1, K / 2048).  bf16 anywhere, in the result or in the
    partial sums of a split reduction, would leave 2^-9 / sqrt(3) = 1.1e-3."""
    torch.manual_seed(0)
    w = torch.randn(N, K, device="cuda").bfloat16()
    for M in (1, 16, 97, 256):
        x = torch.randn(M, K, device="cuda").bfloat16()
        y, ref = _run(x, w, N, torch.float32), _exact(x, w)
        err, bound = float((y.double() - ref).norm() / ref.norm()), 1e-5 * max(1.0, K / 2048)
        assert err <= bound, (M, err)
        assert float((y.bfloat16().double() - ref).norm() / ref.norm()) > 10 * bound          # the bound would see it
