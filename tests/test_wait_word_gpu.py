"""A bounded wait that runs out inside a kernel is reported by the engine whose kernel it was, once, at its next call that waits for the
stream.  The word that the kernels would set is set by the host here."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SPEC = dict(hidden=256, layers=1, heads=4, kv_heads=2, head_dim=64, ffn=576, vocab=1024, rms_eps=1e-5)


def _pair():
    from ssd_b200 import lib as L, synth
    from ssd_b200.runner import ModelSpec, PairRunner
    spec = ModelSpec(**SPEC)
    r = PairRunner(spec, spec, spec_k=2, max_batch=1, block_size=64, max_model_len=640, use_graph=True, use_pdl=True)
    for which, role in ((L.TARGET, "target"), (L.DRAFT, "draft")):
        r.bind_weights(which, synth.generate_weights(spec, {"seed": 3, "alpha": 0.9, "role": role, "o_down_std": 0.05}, torch.device("cuda:0")))
    r.finalize()
    return r


def _calls(r):
    from ssd_b200 import lib as L
    table = list(range(10))
    return {"sampled prompt": lambda: r.prefill(L.TARGET, [5] * 300, table),
            "sampled token": lambda: r.forward_tokens(L.TARGET, [[5]], [300], [table]),
            "step": lambda: r.spec_step([300], [5], [table], [table], [0.0], [0.0]),
            "stage": lambda: r.stage([300], [5], [table], [table], [0.0], [0.0]),
            "fetch": lambda: r.fetch(1),
            "log": lambda: r.resident_log(0)}


def test_reported_by_its_engine_at_every_call_that_waits():
    from ssd_b200 import lib as L
    a, b = _pair(), _pair()
    ca, cb = _calls(a), _calls(b)
    word = a.lib.ssdk_debug_wait_word(a.h)
    for name in ca:
        word[0] = 1
        a.prefill(L.DRAFT, [5] * 300, list(range(10)), want_sample=False)   # does not wait: the report stays
        for other in cb.values():
            other()
        assert word[0] == 1
        with pytest.raises(RuntimeError, match="ran out"):
            ca[name]()
        assert word[0] == 0
        ca[name]()


def test_layered_engine_has_its_own():
    from ssd_b200 import hybrid_bench as hb
    from ssd_b200.hybrid import HybridRunner, random_hybrid_weights
    spec = hb.kefurax_spec(dict(hb.SIZES["s"], layers=1, vocab=512), ("rglru",))
    w = random_hybrid_weights(spec, torch.bfloat16, "cuda:0", seed=3)
    a, b = (HybridRunner(spec, w, max_tokens=64, max_seqs=1, block_size=64, num_blocks=2, n_slots=1, max_model_len=128) for _ in range(2))
    p = _pair()
    a.lib.ssdk_hyb_debug_wait_word(a.h)[0] = 1
    b.forward([([1, 2], 0, 0, [0], [1])])
    for call in _calls(p).values():
        call()
    with pytest.raises(RuntimeError, match="ran out"):
        a.forward([([1, 2], 0, 0, [0], [1])])
    a.forward([([1, 2], 0, 0, [0], [1])])
