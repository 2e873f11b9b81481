"""Logits that the sampler takes to the host on its way: vocabularies around whole 16-byte pieces, results in pinned buffers and (while a caller holds those) in
ordinary memory, plain and replayed steps, against calls that only ask for logits."""
import numpy as np
import pytest
import torch

from tests import kefurax_util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab", [49, 50, 51, 52, 1030, 4099])
def test_logits_of_sampled_rows(tmp_path, vocab):
    from ssd_b200.hybrid import HybridRunner, HybridSpec, load_hybrid_weights
    cfg = U.config([U.rglru(width=24, blocks=2)], width=40, vocab=vocab)
    path = U.write_checkpoint(str(tmp_path / "c"), cfg, U.random_tensors(cfg, 5))
    spec = HybridSpec.from_dir(path)
    make = lambda: HybridRunner(spec, load_hybrid_weights(path, spec, torch.bfloat16, "cuda:0"), dtype="bfloat16", max_tokens=32, max_seqs=3, block_size=16, num_blocks=24,
                                n_slots=3, max_model_len=128)
    a, b = make(), make()
    pages = [list(range(i * 8, (i + 1) * 8)) for i in range(3)]
    held, at = [], [0, 0, 0]
    for step in range(8):
        n = 3 if step % 2 == 0 else 1   # tokens of every sequence: a prompt's portion, then single tokens (the last of them as a graph)
        n = 1 if step > 2 else n
        entries = [([(7 * step + 3 * i + k) % vocab for k in range(n)], at[i], i, pages[i], [n - 1]) for i in range(3)]
        at = [x + n for x in at]
        want = b.forward(entries)[0]
        logits, tokens = a.forward(entries, temps=[0.0, 0.0, 0.0])
        assert np.array_equal(logits, want), step
        rounded = torch.from_numpy(want).to(torch.bfloat16)
        for i, t in enumerate(tokens):   # (the largest rounded logit; of equal ones the first)
            assert t == int((rounded[i] == rounded[i].max()).nonzero()[0]), (step, i)
        held.append((logits, want))
        if step == 4:
            held.clear()
    assert all(np.array_equal(x, y) for x, y in held)   # what a caller holds is not written again
