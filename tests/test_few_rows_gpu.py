"""Calls of few rows: routed experts in narrow tiles against the mma.sync tile, at row counts around a tile and with experts that fill
several; latent decoding at contexts of one key to many tiles per split."""
import numpy as np
import pytest
import torch

from tests import lisenex_util as U
from tests.test_lisenex_gpu import _load, _pages, _tokens

pytestmark = pytest.mark.gpu


def test_experts_in_narrow_tiles(tmp_path, monkeypatch):
    """Same routing, same fp32 products in another order, same roundings to bf16 (the activation and the output rows): two of them, on the
    elements near a rounding edge, 2^-8 each."""
    mlp = U.moe(experts=3, identity=1, top=2, groups=2, keep=2, ff=192, shared_ff=64)
    cfg = U.config([U.latent(heads=2, dim=16, rot_dim=16, vdim=16, kv_rank=48, mlp=mlp)], width=192)
    path = U.write_checkpoint(str(tmp_path / "c"), cfg, U.random_tensors(cfg, 13, correction=1.0))
    runners = []
    for tc in ("1", "0"):
        monkeypatch.setenv("SSDK_HYB_TC_EXPERTS", tc)
        runners.append(_load(path, "bfloat16", max_tokens=128, num_blocks=24))
    for n in (1, 2, 7, 16, 17, 33, 64, 127):
        toks = _tokens(n, cfg["vocab"], n)
        a, b = (r.forward([(toks, 0, 0, _pages(n, 16), list(range(n)))])[0] for r in runners)
        assert np.isfinite(a).all()
        assert U.rel_err(a, b) < 2 * 2.0 ** -8, f"{n} rows"


def test_latent_decoding_at_tile_edges(tmp_path, monkeypatch):
    """The tensor-core form against the CUDA-core one: both round queries and keys to bf16, the first also the probabilities (2^-9 each,
    uncorrelated, so less in their weighted sum) and both the output (2^-9): 2^-8 covers it."""
    cfg = U.config([U.latent(heads=3, dim=16, rot_dim=8, vdim=16, kv_rank=48, scale=1.5)], width=64)
    path = U.write_checkpoint(str(tmp_path / "c"), cfg, U.random_tensors(cfg, 17))
    lens = (1, 31, 32, 33, 64, 65, 97, 129, 300, 6500)
    rows = {}
    for mma in ("1", "0"):
        monkeypatch.setenv("SSDK_HYB_DECODE_MMA", mma)
        r = _load(path, "bfloat16", max_tokens=512, max_seqs=2, block_size=64, num_blocks=104, n_slots=2, max_model_len=6656)
        rows[mma] = []
        for n in lens:
            toks, at = _tokens(n, cfg["vocab"], n), 0
            while at < n - 1:
                k = min(512, n - 1 - at)
                r.forward([(toks[at:at + k], at, 0, _pages(n, 64), [k - 1])])
                at += k
            rows[mma].append(r.forward([(toks[at:], at, 0, _pages(n, 64), [0])])[0][0])
        r.close()
    for n, a, b in zip(lens, rows["1"], rows["0"]):
        assert np.isfinite(a).all()
        assert U.rel_err(a, b) < 2.0 ** -8, f"{n} keys"


def test_gate_far_below_zero(tmp_path, monkeypatch):
    """silu(g) for g around -88, where 1 + e^-g is near fp32's largest number and silu(g) is not zero yet, under an up projection that
    makes it visible.  One nonzero weight per gate and up row and an identity behind them: both forms compute the same numbers."""
    ff = W = 192
    mlp = U.moe(experts=3, identity=1, top=2, groups=2, keep=2, ff=ff, shared_ff=None)
    cfg = U.config([U.latent(heads=2, dim=16, rot_dim=16, vdim=16, kv_rank=48, mlp=mlp)], width=W)
    t = U.random_tensors(cfg, 13, correction=1.0)
    size = torch.logspace(np.log10(60.0), np.log10(200.0), ff // 2)
    for e in range(3):
        gate, up = torch.zeros(ff, W), torch.zeros(ff, W)
        gate[:, 0] = torch.cat([size, -size])
        up[:, 1] = 2.0 ** 117
        t[f"l0.mlp.e{e}.gate"], t[f"l0.mlp.e{e}.up"], t[f"l0.mlp.e{e}.down"] = gate.bfloat16().float(), up, torch.eye(W)
    path = U.write_checkpoint(str(tmp_path / "c"), cfg, t)
    none = U.write_checkpoint(str(tmp_path / "d"), cfg, {k: torch.zeros_like(v) if ".down" in k else v for k, v in t.items()})
    toks, rows = _tokens(16, cfg["vocab"], 5), []
    for tc, p in (("1", path), ("0", path), ("0", none)):
        monkeypatch.setenv("SSDK_HYB_TC_EXPERTS", tc)
        rows.append(_load(p, "bfloat16", max_tokens=64, num_blocks=24).forward([(toks, 0, 0, _pages(16, 16), [0])], residual=True)[2][0])
    size = np.abs(rows[1] - rows[2])
    assert ((size > 1e-4) & (size < 1)).any()   # (what the gates around -88 leave)
    assert np.array_equal(rows[0], rows[1])
