"""Prompts of grouped-query attention on tcgen05 tiles (gqa_prompt_kernel) against 64 bits and the path of separate products and a softmax: one and two maps, head
sizes, groups, windows and kept keys around chunks, constant and learned sinks, output gates, two sequences, portions behind earlier ones, a pool
that holds NaN wherever nothing was stored."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(arch, a):
    U = importlib.import_module(f"tests.{arch}_util")
    layer = U.parallel(left=U.attention(**a), right=U.delta()) if arch == "kefurax" else U.attention(**a)
    return U, U.config([layer], width=64)


@pytest.mark.parametrize("arch,a", [
    ("vegilix", dict(heads=8, kv_heads=2, dim=64, vdim=128, window=100, keep=3, scale=0.25, dims=32)),
    ("vegilix", dict(heads=2, kv_heads=2, dim=64, vdim=64, window=200, keep=70, scale=0.25, dims=16)),
    ("vegilix", dict(heads=16, kv_heads=1, dim=64, vdim=128, window=0, scale=0.1, dims=64)),
    ("kefurax", dict(heads=4, kv_heads=1, dim=128, vdim=128, scale=0.2, dims=64)),
    ("kefurax", dict(heads=4, kv_heads=2, dim=64, vdim=128, scale=1.0, dims=64)),
    ("kokatar", dict(heads=8, kv_heads=1, dim=64, vdim=64, window=130, scale=0.2, dims=32)),
    ("kokatar", dict(heads=4, kv_heads=4, dim=128, vdim=64, window=64, scale=0.2, dims=64)),
    ("kokatar", dict(heads=2, kv_heads=1, dim=64, vdim=128, window=1, scale=0.2, dims=0))])
def test_matches_separate_products(tmp_path, monkeypatch, arch, a):
    """Both round keys, probabilities (2^-9 each) and heads to bf16; what differs is the order of fp32 sums and the point at which a probability is
    rounded, which shows as one unit (2^-8) of a head's entries, and again behind the output projection's rounding and the norm: 2^-6 covers it."""
    from ssd_b200.hybrid import HybridRunner, HybridSpec, load_hybrid_weights
    U, cfg = _model(arch, a)
    tensors = U.random_tensors(cfg, 3)
    path = U.write_checkpoint(str(tmp_path / "c"), cfg, tensors)
    plain = (U if arch == "kefurax" else importlib.import_module(f"tests.{arch}_plain")).PlainModel(cfg, tensors)
    spec = HybridSpec.from_dir(path)
    runners = {}
    for on in ("1", "0"):
        monkeypatch.setenv("SSDK_HYB_GQA_MMA", on)
        r = HybridRunner(spec, load_hybrid_weights(path, spec, torch.bfloat16, "cuda:0"), dtype="bfloat16", max_tokens=1024, max_seqs=3, block_size=64, num_blocks=48,
                         n_slots=3, max_model_len=1024)
        r.cache.view(torch.bfloat16).fill_(float("nan"))
        runners[on] = r
    toks = [torch.randint(0, cfg["vocab"], (n,), generator=torch.Generator().manual_seed(n)).tolist() for n in (700, 321, 193)]
    pages = [list(range(i * 16, (i + 1) * 16))[::-1] for i in range(3)]
    want = [plain.run(t).numpy() for t in toks]
    at, rows = [0, 0, 0], {"1": [], "0": [], "want": []}
    for part in ((2, 128, 64), (255, 1, 65), (63, 129, 1), (380, 63, 63)):   # rows of the three sequences in turn
        entries = [(toks[i][at[i]:at[i] + n], at[i], i, pages[i], list(range(n))) for i, n in enumerate(part)]
        rows["want"] += [want[i][at[i]:at[i] + n] for i, n in enumerate(part)]
        at = [x + n for x, n in zip(at, part)]
        got = {}
        for on, r in runners.items():
            logits, _, residual = r.forward(entries, residual=True)
            got[on] = residual[0]
            rows[on].append(logits)
        assert np.isfinite(got["1"]).all()
        assert U.rel_err(got["1"], got["0"]) < 2.0 ** -6, part
    # all rows against 64 bits: no further off than the separate products, which round a weight once as well (a tenth for the order of sums)
    off = {on: U.rel_err(np.concatenate(rows[on]), np.concatenate(rows["want"])) for on in ("1", "0")}
    assert off["1"] < 2.0 ** -6 and off["1"] <= 1.1 * off["0"], off
