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


# how the scores of a row move along the keys, in units of base 2 per chunk of 64 keys: the running maximum then stays, moves by a little
# less or more than the margin that the kernel tolerates (8), moves at every chunk, or never after the first
SLOPES = {"flat": 0.0, "under": 7.5, "over": 8.5, "steep": 20.0, "falling": -9.0}


@pytest.mark.parametrize("slope", SLOPES)
@pytest.mark.parametrize("heads,kv_heads,hd,batch,q_len,ctx0", [(8, 2, 128, 1, 2003, 0), (4, 4, 64, 2, 300, 129), (16, 1, 64, 1, 261, 1000), (8, 1, 128, 3, 64, 65), (2, 2, 128, 1, 129, 0)])
def test_against_float64(heads, kv_heads, hd, batch, q_len, ctx0, slope):
    """The kernel alone against softmax attention in float64, every output element.  A probability and the output are rounded to bf16 (8
    significant bits: 2^-8 of |p v| and of |o| <= sum p |v| each); the scores (up to 650, sums of 128 fp32 products, truncated at
    2^-23 of the partial sum up to eight times) are off by less than 1e-3 of base 2, a weight by 7e-4: 2^-7 + 2^-10 of sum p |v|."""
    from ssd_b200 import lib as L
    g = torch.Generator(device="cuda").manual_seed(heads * 1000 + q_len)
    G, n = heads // kv_heads, ctx0 + q_len
    scale = hd ** -0.5
    unit = torch.zeros(hd, device="cuda"); unit[3] = 1.0
    q = torch.randn(batch, q_len, heads, hd, generator=g, device="cuda") + 16.0 * unit
    k = torch.randn(batch, n, kv_heads, hd, generator=g, device="cuda")
    k += (torch.arange(n, device="cuda") / 64 * SLOPES[slope] / (16.0 * scale * 1.4427)).view(1, n, 1, 1) * unit
    v = torch.randn(batch, n, kv_heads, hd, generator=g, device="cuda")
    q, k, v = (t.to(torch.bfloat16) for t in (q, k, v))
    bs, pages = 64, -(-n // 64)
    order = torch.randperm(batch * pages + 3, generator=torch.Generator().manual_seed(1))[:batch * pages].to(torch.int32).view(batch, pages)
    tables = torch.cat([order, torch.full((batch, 2), -1, dtype=torch.int32)], 1).cuda().contiguous()
    kc, vc = (torch.full((batch * pages + 3, bs, kv_heads, hd), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    for b in range(batch):
        for j in range(pages):
            m = min(bs, n - j * bs)
            kc[order[b, j], :m], vc[order[b, j], :m] = k[b, j * bs:j * bs + m], v[b, j * bs:j * bs + m]
    lens = torch.full((batch,), n, dtype=torch.int32, device="cuda")
    out = torch.full((batch * q_len, heads * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
    gave_up = torch.zeros(1, dtype=torch.int32).pin_memory()
    L.check(L.load().ssdk_prompt_attn(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), tables.data_ptr(), lens.data_ptr(), out.data_ptr(), batch, q_len, heads,
                                      kv_heads, hd, bs, pages + 2, kc.shape[0], scale, gave_up.data_ptr(), torch.cuda.current_stream().cuda_stream), "ssdk_prompt_attn")
    torch.cuda.synchronize()
    assert gave_up.item() == 0
    out = out.view(batch, q_len, heads, hd).double()
    hidden = torch.arange(n, device="cuda")[None, :] > torch.arange(ctx0, n, device="cuda")[:, None]
    for b in range(batch):
        for h in range(heads):
            s = (q[b, :, h].double() @ k[b, :, h // G].double().T) * scale
            p = torch.softmax(s.masked_fill(hidden, float("-inf")), -1)
            vd = v[b, :, h // G].double()
            bound = (2.0 ** -7 + 2.0 ** -10) * (p @ vd.abs())
            off = (out[b, :, h] - p @ vd).abs() / bound
            assert torch.isfinite(off).all() and off.max().item() < 1, (b, h, off.max().item())
