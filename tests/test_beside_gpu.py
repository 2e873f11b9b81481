"""A decoding step's attention beside its delta rule, on a stream of its own, against the two in order and against sequences that step alone: a score buffer
that holds the fused form's partials, and one that does not (as many sequences as tokens, contexts shorter than a value head), whose attention needs the buffer
that the delta rule's results lie in."""
import numpy as np
import pytest
import torch

from tests import kefurax_util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_len", [64, 128, 1024])
def test_full_batch_of_single_tokens(tmp_path, monkeypatch, max_len):
    """Rows, one at a time or together, go through products with the same operands in another order of sums: a rounding to bf16 moves here and there (2^-9
    of a value, a handful of roundings in a layer): 2^-6."""
    from ssd_b200.hybrid import HybridRunner, HybridSpec, load_hybrid_weights
    n = 8
    layer = U.parallel(left=U.attention(heads=4, kv_heads=2, dim=128, vdim=128, dims=64), right=U.delta(heads=4, kv_heads=2, dim=64, vdim=128, conv=4))
    cfg = U.config([layer, layer], width=64)
    tensors = U.random_tensors(cfg, 7)
    path = U.write_checkpoint(str(tmp_path / "c"), cfg, tensors)
    spec = HybridSpec.from_dir(path)

    def make(decode_attn):
        monkeypatch.setenv("SSDK_HYB_DECODE_ATTN", decode_attn)
        return HybridRunner(spec, load_hybrid_weights(path, spec, torch.bfloat16, "cuda:0"), dtype="bfloat16", max_tokens=n, max_seqs=n, block_size=16,
                            num_blocks=n * max_len // 16, n_slots=n, max_model_len=max_len)
    beside, ordered, alone = make("1"), make("0"), make("1")
    per = max_len // 16
    pages = [list(range(i * per, (i + 1) * per)) for i in range(n)]
    g = torch.Generator().manual_seed(3)
    toks = torch.randint(0, cfg["vocab"], (n, 40), generator=g).tolist()
    for t in range(40):
        entries = [([toks[i][t]], t, i, pages[i], [0]) for i in range(n)]
        a, b = beside.forward(entries)[0], ordered.forward(entries)[0]
        c = np.concatenate([alone.forward([e])[0] for e in entries])
        assert np.isfinite(a).all()
        assert U.rel_err(a, b) < 2.0 ** -6 and U.rel_err(a, c) < 2.0 ** -6, t
    want = np.stack([U.PlainModel(cfg, tensors).run(x).numpy()[-1] for x in toks])
    assert U.rel_err(a, want) < 2.0 ** -5   # (bf16 against float64, two layers of states that carry their roundings along)
