"""Products of up to eight rows straight from the operand registers (gemm_few_kernel) against float64: row counts, columns around a tile of 16 (gated: 8)
and above the resident CTAs, k from one unit of 64 to many per warp, uneven shares of k."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _data(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M * 7919 + N * 31 + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(torch.bfloat16)
    return x, w


def _sums(x, w):
    """The product, and what K fp32 additions of exact products can be off by: K 2^-24 of the sum of magnitudes (truncating units: twice that)."""
    y = x.double() @ w.double().T
    return y, 2 * x.shape[1] * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("M", [1, 2, 5, 8])
@pytest.mark.parametrize("N,K", [(1, 64), (15, 128), (16, 448), (17, 512), (100, 576), (1000, 1024), (2048, 1088), (4736, 2048), (9500, 1024), (96, 4096), (250, 14336)])
def test_linear(M, N, K):
    from ssd_b200 import ops
    x, w = _data(M, N, K)
    y, off = _sums(x, w)
    got = ops.linear(x, w).double()
    bound = off + 2.0 ** -8 * y.abs()   # one rounding to bf16 (2^-9), and the sum may have crossed its edge
    assert ((got - y).abs() <= bound).all()


@pytest.mark.parametrize("M", [1, 3, 8])
@pytest.mark.parametrize("F,K", [(8, 64), (72, 576), (1000, 1024), (5000, 1024), (320, 4160)])
def test_gated(M, F, K):
    """silu(gate) * up of sums rounded to bf16: gate and up may each be a neighbour (2^-8), silu's slope is below 1.1, one more rounding behind."""
    from ssd_b200 import ops
    x, w = _data(M, 2 * F, K)
    y, off = _sums(x, w)
    g, u = y.split(F, 1)
    dg, du = (off + 2.0 ** -8 * y.abs()).split(F, 1)
    silu = g * torch.sigmoid(g)
    bound = 1.1 * dg * u.abs() + du * silu.abs() + 1.1 * dg * du + 2.0 ** -7 * (silu * u).abs() + 1e-6
    assert ((ops.gate_up_silu(x, w).double() - silu * u).abs() <= bound).all()


def test_rows_do_not_follow_from_their_neighbours():
    from ssd_b200 import ops
    x, w = _data(8, 3072, 2048)
    assert torch.equal(ops.linear(x, w)[2:5], ops.linear(x[2:5].contiguous(), w))
