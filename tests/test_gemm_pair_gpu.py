"""The two-CTA GEMM of calls with many rows (gemm_pair_kernel) against the one-CTA kernel it takes over from, at row counts around its
tile edges: dense products, the gated feed-forward's epilogue and the grouped experts."""
import dataclasses

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# Both forms add the same fp32 products (in another order where the one-CTA form splits K) and round the same intermediates to bf16: an
# intermediate differs by one bf16 unit (2^-8) at most, on the elements that lie near a rounding edge; three such steps in a layer.
TOL = 3 * 2.0 ** -8


def _spec(kind):
    from ssd_b200 import hybrid_bench as hb
    z = dict(hb.SIZES["s"], layers=2, vocab=512)
    if kind == "dense":      # gelu-GLU behind a recurrence: output widths 1024, 2048 and 2 x 2048 (gated)
        return hb.kefurax_spec(z, ("rglru",))
    spec = hb.lisenex_spec(dict(z, ff=336))  # routed silu-GLU experts, 336 columns each: a tile's second half is partly empty
    spec.layers = [dataclasses.replace(spec.layers[1], kv_from=-1)]
    return spec


@pytest.mark.parametrize("kind", ["dense", "experts"])
def test_same_as_one_cta_form(monkeypatch, kind):
    from ssd_b200.hybrid import HybridRunner, random_hybrid_weights
    spec = _spec(kind)
    w = random_hybrid_weights(spec, torch.bfloat16, "cuda:0", seed=3)
    runners = []
    for mode in ("0", "2"):
        monkeypatch.setenv("SSDK_HYB_PAIR", mode)
        runners.append(HybridRunner(spec, w, max_tokens=600, max_seqs=1, block_size=64, num_blocks=10, n_slots=1, max_model_len=640))
    for n in (1, 31, 64, 65, 128, 129, 191, 192, 255, 256, 257, 513):
        toks = torch.randint(0, spec.vocab, (n,), generator=torch.Generator().manual_seed(n)).tolist()
        a, b = (r.forward([(toks, 0, 0, list(range(10)), list(range(n)))])[0] for r in runners)
        assert np.isfinite(b).all()
        err = np.sqrt(((a - b) ** 2).mean(-1) / (a ** 2).mean(-1))
        assert err.max() < TOL, f"{kind}, {n} rows: row {err.argmax()} off by {err.max():.2e}"


def test_many_tiles_per_pair(monkeypatch):
    """1999 rows through a gated feed-forward of 6000 columns and a head of 8000: five and four tiles per pair of CTAs on 148 SMs, so that
    the load ring and both accumulators run on from tile to tile, with remainders in rows and columns."""
    from ssd_b200 import hybrid_bench as hb
    from ssd_b200.hybrid import HybridRunner, random_hybrid_weights
    spec = hb.kefurax_spec(dict(hb.SIZES["s"], layers=1, vocab=8000, sff=6000 - 2 * 512), ("rglru",))
    assert spec.layers[0].ff == 6000
    w = random_hybrid_weights(spec, torch.bfloat16, "cuda:0", seed=5)
    toks = torch.randint(0, spec.vocab, (1999,), generator=torch.Generator().manual_seed(5)).tolist()
    out = []
    for mode in ("0", "2"):
        monkeypatch.setenv("SSDK_HYB_PAIR", mode)
        r = HybridRunner(spec, w, max_tokens=2000, max_seqs=1, block_size=64, num_blocks=32, n_slots=1, max_model_len=2048)
        out.append(r.forward([(toks, 0, 0, list(range(32)), list(range(1999)))])[0].copy())
        r.close()
    a, b = out
    err = np.sqrt(((a - b) ** 2).mean(-1) / (a ** 2).mean(-1))
    assert np.isfinite(b).all() and err.max() < TOL, f"row {err.argmax()} off by {err.max():.2e}"
