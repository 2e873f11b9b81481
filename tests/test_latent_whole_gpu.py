"""Latent attention of whole prompts with every head's keys and values made first (gqa_prompt_kernel over [M, heads] rows, products with weights whose output
columns are contiguous) against the oracle and the absorbed form: both head sizes, sequences around tiles of 128 queries and chunks of 64 keys, own and
shared pools, full and low-rank queries, learned sinks, output gates, single tokens behind the prompts."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(which):
    arch, dim, rank = which
    U = importlib.import_module(f"tests.{arch}_util")
    kw = dict(heads=4, dim=dim, rot_dim=64, vdim=dim, kv_rank=rank)
    layers = [U.latent(**kw), U.latent(**kw, kv_from=0)] if arch == "lisenex" else [U.latent(**kw, q_rank=64)]
    return U, U.config(layers, width=128), importlib.import_module(f"tests.{arch}_plain").PlainModel


@pytest.mark.parametrize("which", [("lisenex", 64, 64), ("lisenex", 128, 192), ("pikavik", 128, 128), ("pikavik", 64, 256)])
def test_whole_prompts(tmp_path, which):
    """Against the absorbed form, which a call takes as soon as one sequence does not start in it: keys, values and queries are rounded to bf16 at other
    places (2^-9 of each, a handful of them per layer, two layers): 2^-6."""
    from ssd_b200.hybrid import HybridRunner, HybridSpec, load_hybrid_weights
    U, cfg, plain_type = _model(which)
    tensors = U.random_tensors(cfg, 4)
    path = U.write_checkpoint(str(tmp_path / "c"), cfg, tensors)
    spec = HybridSpec.from_dir(path)
    plain = plain_type(cfg, tensors)
    make = lambda: HybridRunner(spec, load_hybrid_weights(path, spec, torch.bfloat16, "cuda:0"), dtype="bfloat16", max_tokens=1024, max_seqs=4, block_size=16, num_blocks=160,
                                n_slots=4, max_model_len=640)
    a, b = make(), make()
    for lens in ((193, 2), (128, 129, 127), (500, 64, 63), (300,)):
        toks = [torch.randint(0, cfg["vocab"], (n,), generator=torch.Generator().manual_seed(n)).tolist() for n in lens]
        pages = [list(range(i * 40, (i + 1) * 40))[::-1] for i in range(4)]
        entries = [(t, 0, i, pages[i], list(range(len(t)))) for i, t in enumerate(toks)]
        one = a.forward(entries)[0]
        other = b.forward(entries + [(toks[0][:1], 0, 3, pages[3], [0])])[0][:one.shape[0]]   # a single token: no whole prompt
        want = np.concatenate([plain.run(t).numpy() for t in toks])
        assert np.isfinite(one).all()
        assert U.rel_err(one, other) < 2.0 ** -6 and U.rel_err(one, want) < max(2.0 ** -6, 1.3 * U.rel_err(other, want)), (which, lens)
        nxt = [([5], len(t), i, pages[i], [0]) for i, t in enumerate(toks)]
        assert U.rel_err(a.forward(nxt)[0], b.forward(nxt)[0]) < 2.0 ** -6, (which, lens)   # what the pools hold
