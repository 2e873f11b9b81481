"""fp32 products as three bf16 pieces on the tensor cores (gemm_split_kernel) against the float64 oracles, forced on for every product that
it can take, and beside the FMA form: prompts around its tile edges, portions, single tokens, grouped experts, batched heads."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# A product of 2^-24 terms summed over k <= 600 and a handful of products in a row stay below 1e-6 .. 1e-5; a piece left out shows as 2^-16.
TOL = 2e-5


def _model(arch):
    U = importlib.import_module(f"tests.{arch}_util")
    if arch == "vegilix":
        cfg = U.config([U.attention(heads=4, kv_heads=2, dim=16, vdim=24, dims=8, window=40, mlp=U.moe(experts=5, top=2, ff=48, shared_ff=16)),
                        U.retention(heads=2, dim=16, vdim=8, dims=8)], width=600, vocab=64)
        plain = importlib.import_module("tests.vegilix_plain").PlainModel
    else:
        cfg = U.config([U.parallel(left=U.attention(heads=4, kv_heads=2, dim=16, vdim=8, dims=8), right=U.delta(heads=4, kv_heads=2, dim=16, vdim=8), mlp=U.dense(320)),
                        U.rglru(width=48, blocks=2), U.mamba1(inner=64, state=8, dt_rank=8)], width=264, vocab=72)
        plain = U.PlainModel
    return U, cfg, plain


@pytest.mark.parametrize("arch", ["vegilix", "kefurax"])
def test_three_pieces_match_the_oracle(tmp_path, monkeypatch, arch):
    from ssd_b200.hybrid import HybridRunner, HybridSpec, load_hybrid_weights
    U, cfg, plain_type = _model(arch)
    tensors = U.random_tensors(cfg, 1)
    path = U.write_checkpoint(str(tmp_path / "ckpt"), cfg, tensors)
    spec = HybridSpec.from_dir(path)
    w = load_hybrid_weights(path, spec, torch.float32, "cuda:0")
    plain = plain_type(cfg, tensors)
    runners = {}
    for mode in ("0", "2"):
        monkeypatch.setenv("SSDK_HYB_SPLIT", mode)
        runners[mode] = HybridRunner(spec, w, dtype="float32", max_tokens=300, max_seqs=2, block_size=16, num_blocks=40, n_slots=2, max_model_len=320)
    toks = torch.randint(0, cfg["vocab"], (261,), generator=torch.Generator().manual_seed(2)).tolist()
    want = plain.run(toks).numpy()
    pages = list(range(20))
    for cuts in ([261], [128, 129, 1, 1, 2], [31, 33, 65, 127, 5]):
        errs = {}
        for mode, r in runners.items():
            got, at = [], 0
            for n in cuts:
                got.append(r.forward([(toks[at:at + n], at, 1, pages, list(range(n)))])[0])
                at += n
            errs[mode] = U.rel_err(np.concatenate(got), want)
        assert errs["2"] < TOL and errs["2"] < max(1e-6, 1.5 * errs["0"]), (cuts, errs)
