"""draft_stream_kernel inside speculative steps of one to eight sequences (drafts wider than 1024 take it for batches): uneven contexts around a round of keys, ranges of a
context, heads of 64 and 128, rows of one to four slots, fragments from shared memory and straight from the words; against the oracle, teacher-forced on the engine's tokens."""
import pytest
import torch

from tests.test_engine_gpu import EPS, _spec, _to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd,lens,ffn", [
    (64, [30], 2560),                        # one sequence; steps of a slot that are no multiple of four
    (128, [300], 4096),                      # two ranges of keys
    (64, [515, 7], 5120),                    # three ranges for one sequence, one for the other
    (128, [40, 255, 256, 9], 1536),          # contexts that reach a second range within the step
    (64, [40, 12, 3], 8192),                 # four slots a tile, a row too long for shared memory of three tokens
    (64, [300, 3, 64, 128, 31], 6144),       # five: the instance of eight
    (128, [20, 21, 22, 23, 24, 25, 26, 254], 2048),
])
def test_batches_on_the_streaming_draft_match_the_oracle(hd, lens, ffn):
    from oracle.model import ModelCfg, OracleModel, random_weights
    from oracle.spec import SpecSession, check_greedy_step, contiguous_block_tables
    from ssd_b200 import lib as L
    from ssd_b200.runner import PairRunner
    dev = torch.device("cuda:0")
    B, K, bs = len(lens), 4, 64
    mb = (max(lens) + 3 * (K + 1)) // bs + 1
    tc = ModelCfg(hidden=256, layers=1, heads=4, kv_heads=2, head_dim=64, ffn=512, vocab=1024, max_pos=bs * mb)
    dc = ModelCfg(hidden=1280, layers=2, heads=1280 // hd, kv_heads=5, head_dim=hd, ffn=ffn, vocab=1024, max_pos=bs * mb, qk_norm=hd == 128)
    wt, wd = random_weights(tc, 31), random_weights(dc, 32)
    r = PairRunner(_spec(tc), _spec(dc), spec_k=K, max_batch=B, block_size=bs, max_model_len=bs * mb, use_graph=True)
    r.bind_weights(L.TARGET, _to_dev(wt, dev))
    r.bind_weights(L.DRAFT, _to_dev(wd, dev))
    r.finalize()
    g = torch.Generator().manual_seed(7)
    prompts = [torch.randint(0, tc.vocab, (n,), generator=g).tolist() for n in lens]
    bt = contiguous_block_tables(B, mb)
    bts = [bt[b].tolist() for b in range(B)]
    s = SpecSession(OracleModel(tc, wt, B * mb, bs), OracleModel(dc, wd, B * mb, bs), K, mb)
    rec = s.prefill(prompts, [0.0] * B, bt, bt.clone())
    for b in range(B):
        r.prefill(L.TARGET, prompts[b], bts[b])
        r.prefill(L.DRAFT, prompts[b], bts[b], want_sample=False)
    ctx = list(lens)
    for step in range(2):
        n0 = r.launch_count
        toks, nacc, nrec = r.spec_step(ctx, rec, bts, bts, [0.0] * B, [0.0] * B)
        assert r.launch_count - n0 < (K + 1) * 2 * 7, "the draft's forwards are not one launch"
        spec = torch.from_numpy(toks)
        lp_o, lq_o = s.spec_step_forced(spec)
        torch.testing.assert_close(r.logits_q(B).cpu().float(), lq_o.float(), atol=0.08, rtol=0.03)
        hard, _ = check_greedy_step(spec, nacc.tolist(), nrec.tolist(), lp_o, lq_o, EPS)
        assert not hard, f"step {step}: {hard}"
        ctx = [c + int(n) + 1 for c, n in zip(ctx, nacc)]
        rec = nrec.tolist()
        s.advance(nacc.tolist(), rec)
    r.close()
