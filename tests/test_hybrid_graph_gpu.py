"""Decode steps replayed as graphs, and programmatic dependent launch, give the bits of plain launches: every design, contexts that cross
the attention's split edges, greedy and sampled rows, changed batches, and steps without logits or tokens in between."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(spec, w, dtype, monkeypatch, plain):
    from ssd_b200.hybrid import HybridRunner
    monkeypatch.setenv("SSDK_HYB_GRAPH", "0" if plain else "1")
    monkeypatch.setenv("SSDK_HYB_PDL", "0" if plain else "1")
    r = HybridRunner(spec, w, dtype=dtype, max_tokens=256, max_seqs=3, block_size=16, num_blocks=48, n_slots=3, max_model_len=256)
    g = torch.Generator().manual_seed(1)
    tables = [list(range(16 * i, 16 * (i + 1))) for i in range(3)]
    pos = [121, 63, 7]
    out = [r.forward([(torch.randint(0, spec.vocab, (pos[i],), generator=g).tolist(), 0, i, tables[i], [pos[i] - 1]) for i in range(3)])[0]]
    toks = torch.randint(0, spec.vocab, (3,), generator=g).tolist()
    for step in range(14):
        live = [0, 1, 2] if step % 5 else [2, 0]
        temps = [0.0, 0.8, 0.0][:len(live)] if step % 4 != 3 else None
        lg, tk = r.forward([([toks[i]], pos[i], i, tables[i], [0]) for i in live], temps=temps, seed=11)
        out.append(lg)
        for j, i in enumerate(live):
            pos[i] += 1
            toks[i] = tk[j] if tk is not None else int(lg[j].argmax())
        out.append(np.array([toks]))
    count = r.launch_count
    r.close()
    return out, count


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("arch", ["pikavik", "kefurax", "lisenex", "kokatar", "vatolorn", "vegilix"])
def test_same_bits_as_plain_launches(monkeypatch, arch, dtype):
    from ssd_b200 import hybrid_bench as hb
    from ssd_b200.hybrid import random_hybrid_weights
    spec = getattr(hb, arch + "_spec")(dict(hb.SIZES["s"], layers=4, vocab=1000))
    w = random_hybrid_weights(spec, getattr(torch, dtype), "cuda:0", seed=2)
    want, n_plain = _run(spec, w, dtype, monkeypatch, True)
    got, n = _run(spec, w, dtype, monkeypatch, False)
    assert n == n_plain
    for i, (a, b) in enumerate(zip(want, got)):
        assert np.array_equal(a, b), f"output {i}"
