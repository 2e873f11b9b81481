"""Pin the oracle (CPU restatement) against golden vectors produced by the reference's own code
(oracle/gen_golden.py).  CPU only."""
import numpy as np
import pytest
import torch

from oracle import ops, verify as V
from oracle.model import OracleModel
from oracle.spec import SpecSession, check_greedy_step, contiguous_block_tables
from tests.helpers import bf16, load, trace_cfgs, trace_weights, ulp_mismatch_fraction


def test_verify_temp0_matches_reference():
    z = load("verify_t0.npz")
    for c in range(int(z["n_cases"])):
        lp, lq, spec = bf16(z[f"c{c}_lp"]), bf16(z[f"c{c}_lq"]), torch.from_numpy(z[f"c{c}_spec"])
        B = lp.shape[0]
        suf, rec = V.verify(lp, lq, spec, torch.zeros(B), torch.zeros(B))
        assert [len(s) - 1 for s in suf] == z[f"c{c}_nacc"].tolist()
        assert rec == z[f"c{c}_rec"].tolist()
        assert [t for s in suf for t in s] == z[f"c{c}_suffix_flat"].tolist()


def test_verify_ratio_matches_reference():
    """temp>0: same acceptance decisions for the same uniforms; same distributions handed to multinomial."""
    z = load("verify_ratio.npz")
    for c in range(int(z["n_cases"])):
        lp, lq, spec = bf16(z[f"c{c}_lp"]), bf16(z[f"c{c}_lq"]), torch.from_numpy(z[f"c{c}_spec"])
        tt, tq, jit = z[f"c{c}_cfg"].tolist()
        B = lp.shape[0]
        hits = torch.from_numpy(z[f"c{c}_hits"]) if f"c{c}_hits" in z else None
        uni = torch.from_numpy(z[f"c{c}_uni"])
        suf, rec, dbg = V.verify(lp, lq, spec, torch.full((B,), tt), torch.full((B,), tq), hits, bool(jit), uni,
                                 return_debug=True)
        assert [len(s) - 1 for s in suf] == z[f"c{c}_nacc"].tolist(), f"case {c}"
        nd = int(z[f"c{c}_ndist"])
        if tt > 0:
            # reference hands [adj_norm, fallbackDist] (any ratio row) or [fallbackDist] to multinomial
            fallback = torch.from_numpy(z[f"c{c}_dist{nd - 1}"])
            adj = torch.from_numpy(z[f"c{c}_dist0"]) if nd == 2 else None
            for b in range(B):
                got = dbg["recovery_dists"][b]
                n = int(dbg["accept_until"][b])
                K = lq.shape[1]
                ratio_row = bool(jit) or (hits is not None and bool(hits[b]))
                want = adj[b] if (adj is not None and ratio_row and n < K) else fallback[b]
                torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-8)
                # and with multinomial := argmax the reference's recovery is the mode of that distribution
                assert int(want.argmax()) == int(z[f"c{c}_rec_argmax"][b])
        else:
            assert rec == z[f"c{c}_rec_argmax"].tolist()


def test_sampler_greedy_matches_reference():
    z = load("sampler_t0.npz")
    toks = V.sample(bf16(z["logits"]), torch.zeros(4))
    assert toks.tolist() == z["tokens"].tolist()


@pytest.mark.parametrize("tag,compiled", [("compiled", True), ("eager", False)])
def test_layers_match_reference(tag, compiled):
    z = load(f"layers_{tag}.npz")
    x, res, w = bf16(z["norm_x"]), bf16(z["norm_res"]), bf16(z["norm_w"])
    y = ops.rms_norm(x, w, 1e-5, compiled=compiled)
    y2, r2 = ops.rms_norm(x, w, 1e-5, res, compiled=compiled)
    # reduction order inside Inductor differs: allow a vanishing fraction of 1-ulp flips (1.7e-5)
    assert ulp_mismatch_fraction(y, bf16(z["norm_y"])) < 2e-3
    assert ulp_mismatch_fraction(y2, bf16(z["norm_add_y"])) < 2e-3
    assert torch.equal(r2, bf16(z["norm_add_res"]))
    yh = ops.rms_norm(bf16(z["hnorm_x"]), bf16(z["hnorm_w"]), 1e-6, compiled=compiled)
    assert ulp_mismatch_fraction(yh, bf16(z["hnorm_y"])) < 2e-3
    table = ops.rope_table(64, 512, 500000.0)
    assert torch.equal(table, torch.from_numpy(z["rope_table"]))
    pos = torch.from_numpy(z["rope_pos"])
    q, k = bf16(z["rope_q"]), bf16(z["rope_k"])
    qo = ops.apply_rope(q.view(6, 4, 64), pos, table).reshape(6, -1)
    ko = ops.apply_rope(k.view(6, 2, 64), pos, table).reshape(6, -1)
    assert ulp_mismatch_fraction(qo, bf16(z["rope_qo"])) < 2e-3
    assert ulp_mismatch_fraction(ko, bf16(z["rope_ko"])) < 2e-3
    sy = ops.silu_and_mul(bf16(z["silu_x"]), compiled=compiled)
    assert ulp_mismatch_fraction(sy, bf16(z["silu_y"])) < 2e-3


def test_compiled_and_eager_goldens_differ():
    """Guards the claim that the reference *as run* (torch.compile) single-rounds RMSNorm/SiLU*mul."""
    a, b = load("layers_compiled.npz"), load("layers_eager.npz")
    assert ulp_mismatch_fraction(bf16(a["norm_add_y"]), bf16(b["norm_add_y"])) > 0.05
    assert ulp_mismatch_fraction(bf16(a["silu_y"]), bf16(b["silu_y"])) > 0.05
    assert torch.equal(bf16(a["rope_qo"]), bf16(b["rope_qo"]))


@pytest.mark.parametrize("family", ["llama", "qwen"])
def test_sync_sd_trace_matches_reference(family):
    """Whole draft->verify->accept loop against the reference's model classes + Sampler + verify() for 10 steps of
    2 sequences (temp 0), teacher-forced on the reference's tokens: every decision whose top-2 logit margin is
    >= EPS must agree exactly; near-ties may differ (reduction order: Inductor vs this restatement)."""
    EPS = 0.06  # ~2 bf16 ulps at |logit| ~ 4
    z = load(f"trace_{family}.npz")
    tc, dc = trace_cfgs(family, z)
    K, bs, mb = int(z["K"]), int(z["block_size"]), int(z["max_blocks"])
    B = 2
    t = OracleModel(tc, trace_weights(z, "t"), B * mb, bs)
    d = OracleModel(dc, trace_weights(z, "d"), B * mb, bs)
    s = SpecSession(t, d, K, mb)
    bt = contiguous_block_tables(B, mb)
    prompts = [z["prompt0"].tolist(), z["prompt1"].tolist()]
    rec = s.prefill(prompts, [0.0, 0.0], bt, bt.clone())
    assert rec == z["rec0"].tolist()
    n_steps = z["spec"].shape[0]
    soft_total, decisions = 0, 0
    for step in range(n_steps):
        spec = torch.from_numpy(z["spec"][step])
        nacc = z["nacc"][step].tolist()
        nxt = z["spec"][step + 1][:, 0].tolist() if step + 1 < n_steps else z["final_recovery"].tolist()
        assert spec[:, 0].tolist() == s.recovery
        lp, lq = s.spec_step_forced(spec)
        if step == 0:
            torch.testing.assert_close(lp.float(), bf16(z["lp0"]).float(), atol=0.06, rtol=0.02)
            torch.testing.assert_close(lq.float(), bf16(z["lq0"]).float(), atol=0.06, rtol=0.02)
        hard, soft = check_greedy_step(spec, nacc, nxt, lp, lq, EPS)
        assert not hard, f"step {step}: {hard}"
        soft_total += len(soft)
        decisions += B * (K + 1) + sum(nacc)
        s.advance(nacc, nxt)
    assert soft_total <= max(2, decisions // 20), f"{soft_total} near-tie flips in {decisions} decisions"


def test_baseline_config0_plumbing_1b_shapes_on_cpu():
    """Llama-3 1B, autoregressive, greedy, b=1 on CPU: the reference itself cannot
    run on CPU (engine/model_runner.py:88-89 hard-require CUDA), so the plumbing check is the oracle driving the
    Llama-3.2-1B layer shapes (2 of 16 layers, reduced vocab to keep the CPU suite fast) autoregressively and being
    reproduced exactly by its own speculative path (SD == AR)."""
    from oracle.model import ModelCfg, random_weights
    cfg = ModelCfg(hidden=2048, layers=2, heads=32, kv_heads=8, head_dim=64, ffn=8192, vocab=4096, max_pos=512)
    w = random_weights(cfg, 3)
    mb, bs = 1, 256
    ar = SpecSession(OracleModel(cfg, w, mb, bs), None, 0, mb)
    bt = contiguous_block_tables(1, mb)
    prompt = list(range(7, 39))
    ar.prefill([prompt], [0.0], bt, None)
    ar_tokens = []
    for _ in range(12):
        ar_tokens += ar.ar_step()
    K = 3
    sd = SpecSession(OracleModel(cfg, w, mb, bs), OracleModel(cfg, w, mb, bs), K, mb)
    sd.prefill([prompt], [0.0], bt, bt.clone())
    sd_tokens = []
    while len(sd_tokens) < 12:
        suf, *_ = sd.spec_step()
        assert len(suf[0]) == K + 1  # identical draft: everything is accepted
        sd_tokens += suf[0]
    assert sd_tokens[:12] == ar_tokens[:12]


def test_verify_mixed_rows_match_reference():
    """Greedy and sampled rows in one batch, cache-hit gating, K = 1..7: accept counts, suffixes and the recovery rule
    (mode of the distribution the reference hands to multinomial; greedy token on temp-0 rows) match the reference."""
    z = load("verify_mixed.npz")
    for c in range(int(z["n_cases"])):
        lp, lq, spec = bf16(z[f"c{c}_lp"]), bf16(z[f"c{c}_lq"]), torch.from_numpy(z[f"c{c}_spec"])
        tt, tq = torch.from_numpy(z[f"c{c}_tt"]), torch.from_numpy(z[f"c{c}_tq"])
        jit = bool(int(z[f"c{c}_jit"]))
        hits = torch.from_numpy(z[f"c{c}_hits"]) if f"c{c}_hits" in z else None
        uni = torch.from_numpy(z[f"c{c}_uni"])
        suf, rec, dbg = V.verify(lp, lq, spec, tt, tq, hits, jit, uni, return_debug=True)
        assert [len(s) - 1 for s in suf] == z[f"c{c}_nacc"].tolist(), f"case {c}"
        assert [t for s in suf for t in s] == z[f"c{c}_suffix_flat"].tolist(), f"case {c}"
        for b in range(lp.shape[0]):
            want = int(z[f"c{c}_rec_argmax"][b])
            if float(tt[b]) > 0:
                assert int(dbg["recovery_dists"][b].argmax()) == want, f"case {c} row {b}"
            else:
                assert rec[b] == want, f"case {c} row {b}"
