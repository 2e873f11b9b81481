"""Plain decoding (PairRunner.forward_tokens, one token per sequence) of a model as wide as the streaming kernel takes: logits, keys and sampled tokens against the oracle."""
import pytest
import torch

from tests.test_engine_gpu import _spec, _to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,temp", [([0], 0.0), ([300, 1, 63], 0.0), ([64, 5, 255, 256, 257, 2], 0.0), ([33, 70], 0.8)])
def test_one_token_per_sequence_matches_the_oracle(lens, temp):
    from oracle import verify as V
    from oracle.model import ModelCfg, OracleModel, random_weights
    from ssd_b200 import lib as L
    from ssd_b200.runner import PairRunner
    dev = torch.device("cuda:0")
    B, bs = len(lens), 64
    mb = (max(lens) + 4) // bs + 1
    cfg = ModelCfg(hidden=1280, layers=4 if B > 4 else 2, heads=20, kv_heads=5, head_dim=64, ffn=2560, vocab=1024, max_pos=bs * mb)
    w = random_weights(cfg, 33)
    r = PairRunner(_spec(cfg), None, spec_k=0, max_batch=B, block_size=bs, max_model_len=bs * mb)
    r.bind_weights(L.TARGET, _to_dev(w, dev))
    r.finalize()
    model = OracleModel(cfg, w, num_blocks=B * mb, block_size=bs)
    g = torch.Generator().manual_seed(5)
    tables = torch.arange(B * mb, dtype=torch.int32).view(B, mb)

    def slots(b, pos):
        return torch.tensor([int(tables[b][p // bs]) * bs + p % bs for p in pos], dtype=torch.int32)

    for b, n in enumerate(lens):
        if n:
            prompt = torch.randint(0, cfg.vocab, (n,), generator=g)
            r.prefill(L.TARGET, prompt.tolist(), tables[b].tolist(), want_sample=False)
            model.forward(prompt, torch.arange(n), slots(b, range(n)), torch.tensor([n], dtype=torch.int32), tables[b:b + 1], n)
    toks = torch.randint(0, cfg.vocab, (B,), generator=g).tolist()
    n0, step = r.launch_count, r.step_id
    out = r.forward_tokens(L.TARGET, [[t] for t in toks], lens, tables.tolist(), temps=[temp] * B, seed=7)
    assert r.launch_count - n0 <= 2
    got = r.logits_last(B).float().cpu()
    # 0.08 for two layers (as in the other engine tests), 0.05 for the keys of the second; the bf16 roundings of further layers are independent and add in quadrature
    deeper = (cfg.layers / 2) ** 0.5
    for b, n in enumerate(lens):
        h = model.forward(torch.tensor([toks[b]]), torch.tensor([n]), slots(b, [n]), torch.tensor([n + 1], dtype=torch.int32), tables[b:b + 1], 1)
        torch.testing.assert_close(got[b], model.compute_logits(h)[0].float(), atol=0.08 * deeper, rtol=0.03)
    mine = V.sample(r.logits_last(B).cpu(), torch.tensor([temp] * B), 7, step * 16 + 14)
    assert list(out) == mine.tolist()
    kv = r.kv[L.TARGET].float().cpu()
    ref = model.kv_cache.float()
    for b, n in enumerate(lens):
        s = int(slots(b, [n])[0])
        for i in range(2):
            for got_kv, want, atol in zip(kv[i].reshape(cfg.layers, -1, cfg.kv_heads, 64)[:, s], ref[i].reshape(cfg.layers, -1, cfg.kv_heads, 64)[:, s], [0.05] * 2 + [0.05 * deeper] * cfg.layers):
                torch.testing.assert_close(got_kv, want, atol=atol, rtol=0.02)
    r.close()
