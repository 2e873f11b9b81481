"""Attention of prompts in 32 bits, whose products leave out what no row sees (gemm_split_kernel with `see`) and whose softmax leaves its weights as three bf16
pieces, against the float64 oracle: prompts around chunks of 192 (query, head) rows and tiles of 256 keys, above 1024 keys (a block per softmax row), windows
beside kept keys, portions behind earlier ones, two column tiles of values, a latent pool."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# A product of 2^-24 terms summed over k <= 1200 and a handful of products in a row stay below 1e-5; a key left out shows as 1e-3 and more.
TOL = 2e-5


@pytest.mark.parametrize("arch,layer,portions", [
    ("vegilix", dict(heads=4, kv_heads=2, dim=16, vdim=24, dims=8, window=None), ((255, 190), (2, 67), (400, 1))),
    ("vegilix", dict(heads=3, kv_heads=1, dim=64, vdim=264, dims=8, window=None), ((257, 64), (129, 200))),
    ("vegilix", dict(heads=2, kv_heads=1, dim=8, vdim=8, dims=8, window=None), ((1100, 30), (90, 1))),
    ("vegilix", dict(heads=4, kv_heads=2, dim=16, vdim=16, dims=8, window=130, keep=5), ((300, 131), (140, 7))),
    ("kokatar", dict(heads=6, kv_heads=2, dim=16, vdim=8, dims=8, window=513), ((193, 192), (577, 3))),
    ("lisenex", dict(heads=3, dim=16, rot_dim=8, vdim=16, kv_rank=64), ((321, 65), (60, 300)))])
def test_prompts(tmp_path, monkeypatch, arch, layer, portions):
    from ssd_b200.hybrid import HybridRunner, HybridSpec, load_hybrid_weights
    monkeypatch.setenv("SSDK_HYB_SPLIT", "2")
    U = importlib.import_module(f"tests.{arch}_util")
    cfg = U.config([U.latent(**layer) if arch == "lisenex" else U.attention(**layer)], width=64)
    tensors = U.random_tensors(cfg, 5)
    path = U.write_checkpoint(str(tmp_path / "c"), cfg, tensors)
    spec = HybridSpec.from_dir(path)
    plain = importlib.import_module(f"tests.{arch}_plain").PlainModel(cfg, tensors)
    r = HybridRunner(spec, load_hybrid_weights(path, spec, torch.float32, "cuda:0"), dtype="float32", max_tokens=1536, max_seqs=2, block_size=16, num_blocks=160, n_slots=2,
                     max_model_len=1280)
    toks = [torch.randint(0, cfg["vocab"], (sum(p[i] for p in portions),), generator=torch.Generator().manual_seed(i)).tolist() for i in range(2)]
    want = [plain.run(t).numpy() for t in toks]
    pages = [list(range(i * 80, (i + 1) * 80))[::-1] for i in range(2)]
    at = [0, 0]
    for part in portions:
        got, row = r.forward([(toks[i][at[i]:at[i] + n], at[i], i, pages[i], list(range(n))) for i, n in enumerate(part)])[0], 0
        for i, n in enumerate(part):
            assert U.rel_err(got[row:row + n], want[i][at[i]:at[i] + n]) < TOL, (part, i)
            row += n
            at[i] += n
