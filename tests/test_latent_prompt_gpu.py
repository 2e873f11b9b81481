"""Latent attention over prompts: the per-head products on the two-CTA GEMM against the batched tile they take over from, and the softmax
that holds its row in registers at the edges of what it can hold."""
import dataclasses

import numpy as np
import pytest
import torch

from tests import lisenex_util as U
from tests.test_lisenex_gpu import _load, _pages, _tokens

pytestmark = pytest.mark.gpu

# Both forms add the same fp32 products (another order) and round the same intermediates to bf16: an intermediate differs by one bf16 unit
# (2^-8) at most, on the elements near a rounding edge; absorbed query, probabilities and output of a layer make three such steps.
TOL = 3 * 2.0 ** -8


@pytest.mark.parametrize("gate", [False, True], ids=["plain", "gated"])
def test_head_products_same_as_batched_tile(monkeypatch, gate):
    from ssd_b200 import hybrid_bench as hb
    from ssd_b200.hybrid import HybridRunner, random_hybrid_weights
    z = dict(hb.SIZES["s"], layers=2, vocab=512)
    spec = hb.lisenex_spec(z) if gate else hb.pikavik_spec(dict(z, layers=4))
    own = [ly for ly in spec.layers if ly.mixer == "latent_attention"][0]
    spec.layers = [dataclasses.replace(own, kv_from=-1)]
    w = random_hybrid_weights(spec, torch.bfloat16, "cuda:0", seed=4)
    runners = []
    for mode in ("0", "2"):
        monkeypatch.setenv("SSDK_HYB_PAIR", mode)
        runners.append(HybridRunner(spec, w, max_tokens=600, max_seqs=1, block_size=64, num_blocks=10, n_slots=1, max_model_len=640))
    for n in (2, 31, 64, 127, 129, 255, 257, 513):
        toks = torch.randint(0, spec.vocab, (n,), generator=torch.Generator().manual_seed(n)).tolist()
        a, b = (r.forward([(toks, 0, 0, list(range(10)), list(range(n)))])[0] for r in runners)
        assert np.isfinite(b).all()
        err = np.sqrt(((a - b) ** 2).mean(-1) / (a ** 2).mean(-1))
        assert err.max() < TOL, f"{n} rows: row {err.argmax()} off by {err.max():.2e}"


@pytest.mark.parametrize("n", [2, 128, 1023, 1025, 2049, 8191, 8201])
def test_softmax_row_edges(tmp_path, n):
    """The last row of a prompt portion that ends at n keys against the split-context attention of the same token decoded alone: the two
    share nothing between the cache and the output projection.  Probabilities and products are fp32 in both; n of them are added up in
    another order, each within 2^-23 of its value, so the sums are within sqrt(n) 2^-23 of each other, 16x for the layer's few sums."""
    cfg = U.config([U.latent(heads=5, scale=1.5)])
    path = U.write_checkpoint(str(tmp_path / "ckpt"), cfg, U.random_tensors(cfg, 3))
    r = _load(path, max_tokens=512, max_seqs=2, block_size=64, num_blocks=2 * 130, n_slots=2, max_model_len=8320)
    toks = _tokens(n, cfg["vocab"], n)
    rows = []
    for slot, last in ((0, min(3, n)), (1, 1)):   # the portion that ends the prompt: three tokens, or one
        pages, at = _pages(n, 64, 130 * slot), 0
        while at < n - last:
            k = min(512, n - last - at)
            r.forward([(toks[at:at + k], at, slot, pages, [k - 1])])
            at += k
        rows.append(r.forward([(toks[at:], at, slot, pages, [last - 1])])[0][-1])
    assert np.isfinite(rows[0]).all()
    assert U.rel_err(rows[0], rows[1]) < 16 * max(n, 16) ** 0.5 * 2.0 ** -23


def test_softmax_over_infinite_scores(tmp_path):
    """A row whose only visible score is -inf has no softmax (NaN, as inf - inf), like one whose score is +inf; both rows of a prompt of
    two tokens whose keys hold an infinity in an entry that is not rotated."""
    cfg = U.config([U.latent(heads=1, rot_dim=8, dims=4, scale=1.0)])
    t = U.random_tensors(cfg, 3)
    t["l0.mix.dkv"][20 + 6, 0] = float("inf")   # (kv_rank 20, then the key's 8 entries)
    r = _load(U.write_checkpoint(str(tmp_path / "ckpt"), cfg, t), max_tokens=64)
    for tok in range(16):
        rows = r.forward([([tok, 2 * tok + 1], 0, 0, _pages(2, 16), [0, 1])])[0]
        assert np.isnan(rows[0]).all(), tok
