"""Which calls the streaming kernel takes (use_draft_stream, stream_decode in csrc/engine.cu): rows of any length that its slots hold."""
import pytest
import torch

from tests.test_engine_gpu import EPS, _spec, _to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,hd,ffn", [
    (1024, 64, 1280),     # five quarters of a narrow model's usual slot
    (512, 64, 2560),      # two slots of 1280 columns
    (512, 128, 5120),     # four of 1280
    (256, 64, 8192),      # four of 2048
])
def test_narrow_drafts_with_long_or_odd_rows_stream(hidden, hd, ffn):
    from oracle.model import ModelCfg, OracleModel, random_weights
    from oracle.spec import SpecSession, check_greedy_step, contiguous_block_tables
    from ssd_b200 import lib as L
    from ssd_b200.runner import PairRunner
    dev = torch.device("cuda:0")
    K, bs, mb, n = 4, 64, 2, 30
    tc = ModelCfg(hidden=256, layers=1, heads=4, kv_heads=2, head_dim=64, ffn=512, vocab=1024, max_pos=bs * mb)
    dc = ModelCfg(hidden=hidden, layers=2, heads=hidden // hd, kv_heads=2, head_dim=hd, ffn=ffn, vocab=1024, max_pos=bs * mb, qk_norm=hd == 128)
    wt, wd = random_weights(tc, 31), random_weights(dc, 32)
    r = PairRunner(_spec(tc), _spec(dc), spec_k=K, max_batch=1, block_size=bs, max_model_len=bs * mb, use_graph=True)
    r.bind_weights(L.TARGET, _to_dev(wt, dev))
    r.bind_weights(L.DRAFT, _to_dev(wd, dev))
    r.finalize()
    prompt = torch.randint(0, tc.vocab, (n,), generator=torch.Generator().manual_seed(7)).tolist()
    bt = contiguous_block_tables(1, mb)
    table = bt[0].tolist()
    s = SpecSession(OracleModel(tc, wt, mb, bs), OracleModel(dc, wd, mb, bs), K, mb)
    rec = s.prefill([prompt], [0.0], bt, bt.clone())
    r.prefill(L.TARGET, prompt, table)
    r.prefill(L.DRAFT, prompt, table, want_sample=False)
    n0 = r.launch_count
    toks, nacc, nrec = r.spec_step([n], rec, [table], [table], [0.0], [0.0])
    assert r.launch_count - n0 < (K + 1) * 2 * 7, "the draft's forwards are not one launch"
    spec = torch.from_numpy(toks)
    lp_o, lq_o = s.spec_step_forced(spec)
    # bf16 roundings of two layers on logits of unit scale, the bound of the other engine tests
    torch.testing.assert_close(r.logits_q(1).cpu().float(), lq_o.float(), atol=0.08, rtol=0.03)
    hard, _ = check_greedy_step(spec, nacc.tolist(), nrec.tolist(), lp_o, lq_o, EPS)
    assert not hard, hard
    r.close()
