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


@pytest.mark.parametrize("capacity,far", [(512, 440), (4096, 2100)])
def test_lengths_of_the_neighbours_do_not_move_a_sequence(capacity, far):
    """One sequence beside three short or three long ones, in tables of one capacity: the same bits, of a step and of plain decoding, whichever form the capacity picks."""
    from oracle.model import ModelCfg, random_weights
    from ssd_b200 import lib as L
    from ssd_b200.runner import PairRunner
    dev = torch.device("cuda:0")
    B, K, bs, n = 4, 4, 64, 40
    mb = capacity // bs
    tc = ModelCfg(hidden=256, layers=1, heads=4, kv_heads=2, head_dim=64, ffn=512, vocab=1024, max_pos=capacity)
    dc = ModelCfg(hidden=1280, layers=2, heads=20, kv_heads=5, head_dim=64, ffn=2560, vocab=1024, max_pos=capacity)
    wt, wd = _to_dev(random_weights(tc, 31), dev), _to_dev(random_weights(dc, 32), dev)
    tables = [list(range(b * mb, (b + 1) * mb)) for b in range(B)]
    seen = []
    for other in (20, far):
        lens = [n] + [other - 3 * b for b in range(B - 1)]
        r = PairRunner(_spec(tc), _spec(dc), spec_k=K, max_batch=B, block_size=bs, max_model_len=capacity, use_graph=True)
        r.bind_weights(L.TARGET, wt)
        r.bind_weights(L.DRAFT, wd)
        r.finalize()
        g = torch.Generator().manual_seed(9)
        own = torch.randint(0, 1024, (n,), generator=g).tolist()
        for b, m in enumerate(lens):
            prompt = own if b == 0 else torch.randint(0, 1024, (m,), generator=g).tolist()
            for which in (L.TARGET, L.DRAFT):
                r.prefill(which, prompt, tables[b], want_sample=False)
        out = r.forward_tokens(L.DRAFT, [[5 + b] for b in range(B)], lens, tables)
        token, logits = int(out[0]), r.logits_last(B)[0].clone()
        toks, _, _ = r.spec_step(lens, [5 + b for b in range(B)], tables, tables, [0.0] * B, [0.0] * B)
        kv = r.kv[L.DRAFT].reshape(2, dc.layers, -1, dc.kv_heads, dc.head_dim)[:, :, :n + K + 1]
        seen.append((token, logits, torch.as_tensor(toks[0]), r.logits_q(B)[0].clone(), r.logits_p(B)[0].clone(), kv.clone()))
        r.close()
    for a, b in zip(*seen):
        assert a == b if isinstance(a, int) else torch.equal(a, b)
