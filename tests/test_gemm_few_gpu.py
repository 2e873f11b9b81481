"""Products of up to eight rows straight from the operand registers (gemm_few_kernel) against float64: row counts, columns around a tile of 16 (gated: 8)
and above the resident CTAs, k from one unit of 64 to many per warp, uneven shares of k."""
import numpy as np
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


@pytest.mark.parametrize("arch,layer", [
    ("kefurax", dict(type="rglru", width=256, blocks=4)), ("kefurax", dict(type="rglru", width=1280, blocks=2)),
    ("lisenex", dict(heads=3, dim=64, rot_dim=64, vdim=72, kv_rank=64)), ("pikavik", dict(heads=5, dim=128, rot_dim=8, vdim=8, kv_rank=192, q_rank=64))])
def test_heads(tmp_path, arch, layer):
    """Products side by side (the block-diagonal gates of a gated recurrence, latent attention's products per head): a step of 1 to 8 rows against the same
    rows among more than eight, which take the batched tile, and a prompt against the oracle.  Sums in another order move a rounding to bf16 here and there
    (2^-9 of a value, a handful of roundings in a layer): 2^-6."""
    import importlib
    from ssd_b200.hybrid import HybridRunner, HybridSpec, load_hybrid_weights
    U = importlib.import_module(f"tests.{arch}_util")
    layer = dict(layer)
    cfg = U.config([U.rglru(**layer) if layer.pop("type", "") == "rglru" else U.latent(**layer)], width=64)
    tensors = U.random_tensors(cfg, 3)
    path = U.write_checkpoint(str(tmp_path / "c"), cfg, tensors)
    spec = HybridSpec.from_dir(path)
    plain = (U if arch == "kefurax" else importlib.import_module(f"tests.{arch}_plain")).PlainModel(cfg, tensors)
    make = lambda: HybridRunner(spec, load_hybrid_weights(path, spec, torch.bfloat16, "cuda:0"), dtype="bfloat16", max_tokens=512, max_seqs=9, block_size=16, num_blocks=72,
                                n_slots=9, max_model_len=128)
    a, b = make(), make()
    toks = [torch.randint(0, cfg["vocab"], (n,), generator=torch.Generator().manual_seed(n)).tolist() for n in (100, 3, 17, 1, 64, 2, 31, 9, 5)]
    pages = [list(range(i * 8, (i + 1) * 8)) for i in range(9)]
    for r in (a, b):
        first = r.forward([(t, 0, i, pages[i], list(range(len(t)))) for i, t in enumerate(toks)])[0]
        assert U.rel_err(first[:100], plain.run(toks[0]).numpy()) < 2.0 ** -5   # (bf16 against float64)
    at = [len(t) for t in toks]
    for n in (1, 2, 5, 8):
        few = a.forward([([7 + n], at[i], i, pages[i], [0]) for i in range(n)])[0]
        rest = [([3], at[i], i, pages[i], [0]) for i in range(n, 9)]
        many = b.forward([([7 + n], at[i], i, pages[i], [0]) for i in range(n)] + rest)[0]
        assert np.isfinite(few).all() and U.rel_err(few, many[:n]) < 2.0 ** -6, n
        for i in range(n, 9):   # (the other rows in portions of one, so that both hold the same)
            a.forward([([3], at[i], i, pages[i], [0])])
        at = [x + 1 for x in at]
