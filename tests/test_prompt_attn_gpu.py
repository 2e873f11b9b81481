"""Attention of long prompt passes on tcgen05 (prompt_attn_kernel) against the mma.sync tiles it takes over from: head sizes and query
heads per key head, row counts around its tiles and chunks, earlier context, a cache that holds NaN wherever nothing was stored."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# Both round probabilities and outputs to bf16 and add fp32 products in another order: an output differs by one unit (2^-8) near a rounding
# edge, in each of two layers, and the residual stream and the logits round it on: four such steps.
TOL = 4 * 2.0 ** -8


def _runner(heads, kv_heads, hd, batch=2):
    from ssd_b200 import lib as L, synth
    from ssd_b200.runner import ModelSpec, PairRunner
    spec = ModelSpec(hidden=256, layers=2, heads=heads, kv_heads=kv_heads, head_dim=hd, ffn=576, vocab=1024, rms_eps=1e-5)
    r = PairRunner(spec, None, spec_k=0, max_batch=batch, block_size=64, max_model_len=2560, use_graph=False, use_pdl=True)
    w = synth.generate_weights(spec, {"seed": 3, "alpha": 0.9, "role": "target", "o_down_std": 0.05}, torch.device("cuda:0"))
    r.bind_weights(L.TARGET, w)
    r.finalize()
    r.kv[L.TARGET].fill_(float("nan"))
    return r


@pytest.mark.parametrize("heads,kv_heads,hd", [(4, 2, 64), (8, 2, 128), (2, 2, 64), (16, 1, 128), (8, 1, 64)])
def test_matches_mma_tiles(monkeypatch, heads, kv_heads, hd):
    from ssd_b200 import lib as L
    runners = []
    for on in ("0", "1"):
        monkeypatch.setenv("SSDK_PROMPT_ATTN", on)
        runners.append(_runner(heads, kv_heads, hd))
    pages = list(range(40))
    for n in (257, 319, 320, 321, 1000, 2047, 2048, 2049, 2400):
        toks = torch.randint(0, 1024, (n,), generator=torch.Generator().manual_seed(n)).tolist()
        out = []
        for r in runners:
            r.prefill(L.TARGET, toks, pages)
            out.append((r.logits_last(1).float().clone(), r.kv[L.TARGET][1, 1, :40].flatten(0, 1)[:n].float().clone()))
        (la, ka), (lb, kb) = out
        assert torch.isfinite(lb).all() and torch.isfinite(kb).all()
        assert ((la - lb).norm() / la.norm()).item() < TOL, n
        assert ((ka - kb).norm(dim=(-1, -2)) / ka.norm(dim=(-1, -2))).max().item() < 2 * TOL, n   # layer 2's values, row by row


def test_several_sequences_and_earlier_context(monkeypatch):
    from ssd_b200 import lib as L
    g = torch.Generator().manual_seed(6)
    prompts = [torch.randint(0, 1024, (n,), generator=g).tolist() for n in (1500, 611)]
    pages = [list(range(40)), list(range(40, 80))]
    got = []
    for on in ("0", "1"):
        monkeypatch.setenv("SSDK_PROMPT_ATTN", on)
        r = _runner(8, 2, 128)
        for p, t, k in zip(prompts, pages, (777, 100)):
            r.prefill(L.TARGET, p[:k], t)
        got.append((r.prefill_many(L.TARGET, prompts, pages, [777, 100]), r.logits_last(1).float().clone()))
    assert got[0][0] == got[1][0]
    assert ((got[0][1] - got[1][1]).norm() / got[0][1].norm()).item() < TOL
