"""Prompt passes of more than 256 rows (gemm_pair_kernel, one slab per product) against passes of 64 rows: logits of the last row, the
cache, several prompts in a pass, and the calls that stay refused."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# bf16 activations through two layers: both forms round the same intermediates, sums over K in another order (split-K) move some of
# them by one unit of 2^-8
TOL = 4 * 2.0 ** -8


def _runner(batch=2):
    from ssd_b200 import lib as L, synth
    from ssd_b200.runner import ModelSpec, PairRunner
    spec = ModelSpec(hidden=256, layers=2, heads=4, kv_heads=2, head_dim=64, ffn=576, vocab=1024, rms_eps=1e-5)
    r = PairRunner(spec, None, spec_k=0, max_batch=batch, block_size=64, max_model_len=2560, use_graph=False, use_pdl=True)
    w = synth.generate_weights(spec, {"seed": 3, "alpha": 0.9, "role": "target", "o_down_std": 0.05}, torch.device("cuda:0"))
    r.bind_weights(L.TARGET, w)
    r.finalize()
    return r


@pytest.mark.parametrize("n", [255, 256, 257, 320, 449, 2049])
def test_long_pass_matches_short_ones(n):
    from ssd_b200 import lib as L
    r = _runner()
    toks = torch.randint(0, 1024, (n,), generator=torch.Generator().manual_seed(n)).tolist()
    a_pages, b_pages = list(range(40)), list(range(40, 80))
    ta = r.prefill(L.TARGET, toks, a_pages, chunk=64)
    la = r.logits_last(1).float()
    tb = r.prefill(L.TARGET, toks, b_pages)
    lb = r.logits_last(1).float()
    assert ta == tb
    assert ((la - lb).norm() / la.norm()).item() < TOL
    ka, kb = (r.kv[L.TARGET][:, :, s:s + 40].flatten(2, 3)[:, :, :n].float() for s in (0, 40))
    assert ((ka - kb).norm() / ka.norm()).item() < TOL


def test_several_prompts_in_a_pass():
    from ssd_b200 import lib as L
    r = _runner()
    g = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, 1024, (n,), generator=g).tolist() for n in (700, 411)]
    pages = [list(range(40)), list(range(40, 80))]
    want = [r.prefill(L.TARGET, p, t, chunk=64) for p, t in zip(prompts, pages)]
    assert r.prefill_many(L.TARGET, prompts, pages, [0, 0]) == want


def test_refused_as_before():
    from ssd_b200 import lib as L
    r = _runner()
    with pytest.raises(RuntimeError):
        r.forward_tokens(L.TARGET, [[1] * 257], [0], [list(range(40))])
    with pytest.raises(RuntimeError):
        r.prefill(L.TARGET, [1] * 600, list(range(40)), chunk=512)


@pytest.mark.parametrize("hidden,hd,qk_norm", [(4352, 64, False), (256, 128, True), (4096, 64, True)])
def test_row_forms(hidden, hd, qk_norm):
    """Norms and rotation of long passes (bf16 products, one or two slices of a row per thread, head norms) against short ones."""
    from ssd_b200 import lib as L, synth
    from ssd_b200.runner import ModelSpec, PairRunner
    spec = ModelSpec(hidden=hidden, layers=1, heads=4, kv_heads=2, head_dim=hd, ffn=576, vocab=1024, rms_eps=1e-5, qk_norm=qk_norm)
    r = PairRunner(spec, None, spec_k=0, max_batch=2, block_size=64, max_model_len=640, use_graph=False, use_pdl=True)
    w = synth.generate_weights(spec, {"seed": 4, "alpha": 0.9, "role": "target", "o_down_std": 0.05}, torch.device("cuda:0"))
    r.bind_weights(L.TARGET, w)
    r.finalize()
    toks = torch.randint(0, 1024, (301,), generator=torch.Generator().manual_seed(hidden)).tolist()
    r.prefill(L.TARGET, toks, list(range(10)), chunk=64)
    la = r.logits_last(1).float().clone()
    r.prefill(L.TARGET, toks, list(range(10, 20)))
    lb = r.logits_last(1).float()
    assert ((la - lb).norm() / la.norm()).item() < TOL
    ka, kb = (r.kv[L.TARGET][:, 0, s:s + 10].flatten(1, 2)[:, :301].float() for s in (0, 10))
    assert ((ka - kb).norm() / ka.norm()).item() < TOL


def test_sampled_prompts_draw_as_in_short_passes():
    """Flat logits under a high temperature: a token is decided by its random numbers, so that equal tokens mean equal draws."""
    from ssd_b200 import lib as L
    g = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, 1024, (n,), generator=g).tolist() for n in (700, 300, 300, 411, 90)]
    pages = [list(range(12 * i, 12 * (i + 1))) for i in range(5)]
    got = []
    for kw in ({"chunk": 256}, {}):
        r = _runner(batch=5)
        first = r.prefill_many(L.TARGET, prompts, pages, [0] * 5, [50.0, 0.0, 50.0, 50.0, 50.0], seed=9, **kw)
        got.append((first, r.forward_tokens(L.TARGET, [[t] for t in first], [len(p) for p in prompts], pages, [50.0] * 5, seed=9), r.step_id))
    assert got[0] == got[1]


def test_many_tiles_per_pair():
    """Projections of 6144 columns and a gated feed-forward of 6016 over 2003 rows: up to three and six tiles per pair of CTAs on 148 SMs."""
    from ssd_b200 import lib as L, synth
    from ssd_b200.runner import ModelSpec, PairRunner
    spec = ModelSpec(hidden=2048, layers=1, heads=64, kv_heads=16, head_dim=64, ffn=6016, vocab=1024, rms_eps=1e-5)
    r = PairRunner(spec, None, spec_k=0, max_batch=2, block_size=64, max_model_len=2048, use_graph=False, use_pdl=True)
    w = synth.generate_weights(spec, {"seed": 4, "alpha": 0.9, "role": "target", "o_down_std": 0.05}, torch.device("cuda:0"))
    r.bind_weights(L.TARGET, w)
    r.finalize()
    toks = torch.randint(0, 1024, (2003,), generator=torch.Generator().manual_seed(8)).tolist()
    r.prefill(L.TARGET, toks, list(range(32)), chunk=64)
    la = r.logits_last(1).float().clone()
    r.prefill(L.TARGET, toks, list(range(32, 64)))
    lb = r.logits_last(1).float()
    assert ((la - lb).norm() / la.norm()).item() < TOL
    ka, kb = (r.kv[L.TARGET][:, 0, s:s + 32].flatten(1, 2)[:, :2003].float() for s in (0, 32))
    assert ((ka - kb).norm(dim=(-1, -2)) / ka.norm(dim=(-1, -2))).max().item() < TOL   # every row's keys and values
