"""The streaming kernel over contexts of which a CTA's range takes more than one round of keys (256), tables of more pages than it copies to shared memory (32), tables that do not name
every page, and draws of a batch inside the launch: plain decoding and drafts against the oracle."""
import pytest
import torch

from tests.test_engine_gpu import _spec, _to_dev

pytestmark = pytest.mark.gpu


def _decode(hd, kv_heads, lens, bs, unnamed=()):
    """One token for each of the sequences, behind random keys and values; unnamed: (sequence, entry) pairs of the tables that are -1."""
    from oracle.model import ModelCfg, OracleModel, random_weights
    from ssd_b200 import lib as L
    from ssd_b200.runner import PairRunner
    B = len(lens)
    mb = max(lens) // bs + 1
    cfg = ModelCfg(hidden=1280, layers=4 if B > 4 else 2, heads=1280 // hd, kv_heads=kv_heads, head_dim=hd, ffn=2560, vocab=1024, max_pos=bs * mb)
    w = random_weights(cfg, 33)
    r = PairRunner(_spec(cfg), None, spec_k=0, max_batch=B, block_size=bs, max_model_len=bs * mb)
    r.bind_weights(L.TARGET, _to_dev(w, torch.device("cuda:0")))
    r.finalize()
    model = OracleModel(cfg, w, num_blocks=B * mb, block_size=bs)
    g = torch.Generator().manual_seed(5)
    tables = torch.randperm(B * mb, generator=g).to(torch.int32).view(B, mb)
    model.kv_cache.copy_(torch.randn(model.kv_cache.shape, generator=g))
    r.kv[L.TARGET].copy_(model.kv_cache)
    given = tables.clone()
    for b, i in unnamed:   # the oracle reads a page of zeros there, the kernel one that holds something else
        given[b, i] = -1
        model.kv_cache[:, :, int(tables[b, i])] = 0
    toks = torch.randint(0, cfg.vocab, (B,), generator=g).tolist()
    n0 = r.launch_count
    r.forward_tokens(L.TARGET, [[t] for t in toks], list(lens), given.tolist())
    assert r.launch_count - n0 <= 2, "not one launch and the sampler"
    got, kv = r.logits_last(B).float().cpu(), r.kv[L.TARGET].float().cpu().reshape(2, cfg.layers, -1, kv_heads, hd)
    for b, n in enumerate(lens):
        page = int(given[b, n // bs])
        slot = torch.tensor([page * bs + n % bs if page >= 0 else -1], dtype=torch.int32)
        h = model.forward(torch.tensor([toks[b]]), torch.tensor([n]), slot, torch.tensor([n + 1], dtype=torch.int32), tables[b:b + 1], 1)
        # 0.08 for two layers, as in the other engine tests; the bf16 roundings of further layers are independent and add in quadrature.  Keys and values of the first two layers 0.05
        torch.testing.assert_close(got[b], model.compute_logits(h)[0].float(), atol=0.08 * (cfg.layers / 2) ** 0.5, rtol=0.03)
        if page >= 0:
            ref = model.kv_cache.float().reshape(2, cfg.layers, -1, kv_heads, hd)[:, :2, int(slot)]
            torch.testing.assert_close(kv[:, :2, int(slot)], ref, atol=0.05, rtol=0.02)
    r.close()


@pytest.mark.parametrize("hd,kv_heads,lens,bs", [
    (64, 20, [2500], 64),                                     # seven ranges of 384
    (64, 20, [700, 30, 513, 257], 16),                        # one range each, up to three rounds; 44 pages, not of whole 32 keys
    (64, 20, [400, 3, 257, 300, 20, 31, 256, 63], 64),        # more units than CTAs
    (128, 10, [4000], 64),                                    # fourteen ranges of 288; 63 pages
    (128, 10, [900, 800, 17, 769], 16),                       # three ranges, the longest of 320
    (128, 10, [400, 3, 290, 300, 20, 31, 256, 63], 64),
])
def test_ranges_of_several_rounds_match_the_oracle(hd, kv_heads, lens, bs):
    _decode(hd, kv_heads, lens, bs)


@pytest.mark.parametrize("hd,kv_heads,lens,bs,unnamed", [
    (64, 5, [0], 64, [(0, 0)]),
    (64, 5, [70, 600, 200], 64, [(0, 0), (1, 3), (1, 9), (2, 3)]),   # a first page, one inside, the new tokens' own
    (128, 5, [0, 300], 16, [(0, 0), (1, 1), (1, 18)]),
])
def test_pages_that_a_table_does_not_name_are_zeros(hd, kv_heads, lens, bs, unnamed):
    _decode(hd, kv_heads, lens, bs, unnamed)


@pytest.mark.parametrize("hd,B", [(64, 3), (128, 4), (64, 7)])
def test_draws_of_a_batch_are_the_samplers(hd, B):
    """A draft's tokens are what the sampler's rule makes of the launch's own logits, with the row's own random numbers; a temperature of zero beside others."""
    from oracle import verify as V
    from oracle.model import ModelCfg, random_weights
    from ssd_b200 import lib as L
    from ssd_b200.runner import PairRunner
    K, bs, mb, dev = 4, 64, 2, torch.device("cuda:0")
    tc = ModelCfg(hidden=256, layers=1, heads=4, kv_heads=2, head_dim=64, ffn=512, vocab=1024, max_pos=bs * mb)
    dc = ModelCfg(hidden=1280, layers=2, heads=1280 // hd, kv_heads=5, head_dim=hd, ffn=2560, vocab=1024, max_pos=bs * mb)
    r = PairRunner(_spec(tc), _spec(dc), spec_k=K, max_batch=B, block_size=bs, max_model_len=bs * mb, use_graph=True)
    r.bind_weights(L.TARGET, _to_dev(random_weights(tc, 31), dev))
    r.bind_weights(L.DRAFT, _to_dev(random_weights(dc, 32), dev))
    r.finalize()
    tables = [[2 * b, 2 * b + 1] for b in range(B)]
    temps = [0.7 + 0.1 * b if b != 1 else 0.0 for b in range(B)]
    for which in (L.TARGET, L.DRAFT):
        r.kv[which].normal_(generator=torch.Generator(device=dev).manual_seed(3))
    for seed in (11, 12):
        step, n0 = r.step_id, r.launch_count
        toks, _, _ = r.spec_step([20 + b for b in range(B)], [7 * b for b in range(B)], tables, tables, [1.0] * B, temps, seed=seed)
        assert r.launch_count - n0 < (K + 1) * 2 * 7, "the draft's forwards are not one launch"
        logits = r.logits_q(B).cpu()
        for k in range(K):
            assert toks[:, k + 1].tolist() == V.sample(logits[:, k], torch.tensor(temps), seed, step * 16 + k).tolist(), (seed, k)
    r.close()
