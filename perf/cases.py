"""Measured cases: what a program that serves models with this package has it do, through its public entry points.

Kinds (key "kind" of a case)
    step       one speculative step of a target / draft pair (PairRunner.spec_step), greedy
    prefill    one prompt through a dense decoder (PairRunner.prefill)
    decode     one token for each of a batch of sequences of a dense decoder (PairRunner.forward_tokens)
    mlp        norm, gate|up with SiLU, down projection of one decoder layer (ops.rms_norm, gate_up_silu, linear)
    attention  rotation, cache write and paged attention of one decoder layer (ops.rope_store_kv, paged_attention)
    hybrid     prompts or single tokens through a stack of layered models (HybridRunner.forward)

Model sizes are those of ssd_b200.synth.SHAPES and ssd_b200.hybrid_bench.SIZES; depths are cut so that a rounding in one
layer does not travel through dozens.  Weights and inputs come from the seed alone.  Heads of the dense pairs are a permutation of
the embedding (the draft's agrees with the target's on 85 % of the tokens), so that greedy choices have wide margins while every
layer still moves the logits."""
from __future__ import annotations

import math

import numpy as np
import torch

from ssd_b200 import hybrid_bench, ops
from ssd_b200 import lib as L
from ssd_b200.hybrid import HybridRunner
from ssd_b200.runner import ModelSpec, PairRunner
from ssd_b200.synth import SHAPES

DEV = "cuda:0"
F64 = torch.float64
PAIRS = {"llama": ("llama-3.1-8b", "llama-3.2-1b"), "qwen": ("qwen3-32b", "qwen3-0.6b")}


def listed():
    return [
        # one user of the 8B + 1B pair: the step that decoding repeats
        {"name": "step_llama_b1", "kind": "step", "pair": "llama", "layers": 32, "draft_layers": 16, "k": 6, "batch": 1, "ctx": 203},
        # four users of the Qwen pair with longer, uneven contexts (draft and target kernel by kernel)
        {"name": "step_qwen_b4", "kind": "step", "pair": "qwen", "layers": 4, "draft_layers": 28, "k": 4, "batch": 4, "ctx": 1500},
        # a long prompt of an odd length
        {"name": "prefill_llama", "kind": "prefill", "shape": "llama-3.1-8b", "layers": 4, "tokens": 2003},
        # plain decoding of sixteen users with contexts up to 4096
        {"name": "decode_llama_b16", "kind": "decode", "shape": "llama-3.1-8b", "layers": 4, "batch": 16, "ctx": 4000},
        # a 70B layer's feed-forward over the seven rows that a step verifies
        {"name": "mlp_70b_verify", "kind": "mlp", "shape": "llama-3.1-70b", "rows": 7},
        # a 70B layer's attention for eight long sequences of seven rows each
        {"name": "attention_70b_long", "kind": "attention", "shape": "llama-3.1-70b", "batch": 8, "rows": 7, "ctx": 8000},
        # layered models: the smallest call there is, one token of one sequence
        {"name": "kefurax_decode_one", "kind": "hybrid", "arch": "kefurax", "size": "s", "layers": 4, "dtype": "bfloat16", "batch": 1, "tokens": 1, "ctx": 300},
        # one prompt as long as the benchmark's, attention + delta rule, selective scan and diagonal recurrence
        {"name": "kefurax_prefill", "kind": "hybrid", "arch": "kefurax", "size": "m", "layers": 4, "dtype": "bfloat16", "batch": 1, "tokens": 2048, "ctx": 0},
        # three uneven prompts in one call, latent attention and routed experts
        {"name": "lisenex_prefill_ragged", "kind": "hybrid", "arch": "lisenex", "size": "m", "layers": 1, "dtype": "bfloat16", "batch": 3, "tokens": 1000, "ctx": 0},
        # eight decoding users, latent attention and routed experts
        {"name": "lisenex_decode_b8", "kind": "hybrid", "arch": "lisenex", "size": "m", "layers": 1, "dtype": "bfloat16", "batch": 8, "tokens": 1, "ctx": 2040},
        # one prompt through windowed differential attention and routed experts
        {"name": "vegilix_prefill", "kind": "hybrid", "arch": "vegilix", "size": "m", "layers": 1, "dtype": "bfloat16", "batch": 1, "tokens": 2001, "ctx": 0},
        # the exact mode: the same design in 32 bits
        {"name": "vegilix_prefill_fp32", "kind": "hybrid", "arch": "vegilix", "size": "m", "layers": 1, "dtype": "float32", "batch": 1, "tokens": 1000, "ctx": 0},
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.99))))))

    kind = rng.choice(["step", "prefill", "decode", "mlp", "attention"] + 5 * ["hybrid"])
    if kind == "step":
        pair = rng.choice(["llama", "qwen"])
        return {"kind": kind, "pair": pair, "layers": rng.randint(2, 8), "draft_layers": rng.randint(4, 16), "k": rng.randint(2, 7),
                "batch": rng.choice([1, 1, 2, 3, 5, 8]), "ctx": log(60, 2000)}
    if kind == "prefill":
        return {"kind": kind, "shape": rng.choice(["llama-3.2-1b", "llama-3.1-8b", "qwen3-0.6b"]), "layers": rng.randint(2, 4), "tokens": log(40, 2000)}
    if kind == "decode":
        return {"kind": kind, "shape": rng.choice(["llama-3.2-1b", "llama-3.1-8b", "qwen3-32b"]), "layers": rng.randint(2, 4), "batch": log(1, 32), "ctx": log(100, 4000)}
    if kind == "mlp":
        return {"kind": kind, "shape": rng.choice(["llama-3.1-70b", "llama-3.1-8b", "qwen3-32b", "llama-3.2-1b"]), "rows": log(1, 64)}
    if kind == "attention":
        rows = rng.choice([1, 1, 3, 5, 7, 8])
        return {"kind": kind, "shape": rng.choice(["llama-3.1-70b", "llama-3.2-1b", "qwen3-32b"]), "batch": log(1, 16), "rows": rows, "ctx": log(60, 8000)}
    arch, size, dtype = rng.choice(["kefurax", "lisenex", "vegilix", "vegilix_retention"]), rng.choice(["s", "m"]), rng.choice(4 * ["bfloat16"] + ["float32"])
    layers = rng.randint(1, 4) if arch == "kefurax" else 1
    if rng.random() < 0.5:
        return {"kind": kind, "arch": arch, "size": size, "layers": layers, "dtype": dtype, "batch": log(1, 8), "tokens": 1, "ctx": log(40, 2000)}
    most = 2048 if dtype == "bfloat16" else 1000 // layers
    batch = rng.choice([1, 1, 2, 3])
    return {"kind": kind, "arch": arch, "size": size, "layers": layers, "dtype": dtype, "batch": batch, "tokens": log(24, most // batch), "ctx": 0}


def ragged(n, batch):
    """Uneven lengths up to n, the first the longest."""
    return [max(1, n - (i * n) // (2 * batch) - 3 * (i > 0)) for i in range(batch)]


def make_gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(seed * 1000003 + salt)


# ------------------------------------------------------------------------------------------------ dense decoders
def model_spec(shape, layers):
    h, _, H, KV, hd, ffn, V, eps, theta, mtype, _ = SHAPES[shape]
    return ModelSpec(hidden=h, layers=layers, heads=H, kv_heads=KV, head_dim=hd, ffn=ffn, vocab=V, rms_eps=eps, rope_theta=theta, qk_norm=mtype == "qwen3")


def normal(g, std, *shape):
    out = torch.empty(*shape, dtype=torch.bfloat16, device=DEV)
    step = max(1, (1 << 27) // max(1, math.prod(shape[1:])))
    for r in range(0, shape[0], step):
        n = min(step, shape[0] - r)
        out[r:r + n] = torch.randn(n, *shape[1:], generator=g, device=DEV) * std
    return out


def successors(vocab, seed):
    """Next token of every token: the target's and the draft's map, which agree on 85 % of the tokens."""
    g = make_gen(seed, 5)
    nxt_t = torch.randperm(vocab, generator=g, device=DEV)
    off = (torch.rand(vocab, generator=g, device=DEV) > 0.85).nonzero().squeeze(1)
    nxt_d = nxt_t.clone()
    nxt_d[off] = nxt_t[torch.roll(off, -1)]
    return nxt_t, nxt_d


def dense_weights(spec, seed, role):
    g = make_gen(seed, 11 if role == "target" else 12)
    d, hd, H, KV, F = spec.hidden, spec.head_dim, spec.heads, spec.kv_heads, spec.ffn
    embed = normal(g, 1.0, spec.vocab, d)
    nxt = successors(spec.vocab, seed)[0 if role == "target" else 1]
    head = torch.empty_like(embed)
    head[nxt] = embed
    out_std = 0.02 / math.sqrt(2 * spec.layers)   # the layers together move the residual stream by about the embedding's size
    w = {"embed": embed, "lm_head": head, "final_norm": 1 + normal(g, 0.1, d), "layers": []}
    for _ in range(spec.layers):
        lw = {"input_norm": 1 + normal(g, 0.1, d), "post_norm": 1 + normal(g, 0.1, d), "qkv": normal(g, 0.02, (H + 2 * KV) * hd, d),
              "o": normal(g, out_std, d, H * hd), "gate_up": normal(g, 0.02, 2 * F, d), "down": normal(g, out_std, d, F)}
        if spec.qk_norm:
            lw["q_norm"], lw["k_norm"] = 1 + normal(g, 0.1, hd), 1 + normal(g, 0.1, hd)
        w["layers"].append(lw)
    return w


def dense_setup(case, seed):
    """Specs, first context positions, tokens in hand, cached keys and values of a dense case."""
    kind = case["kind"]
    if kind == "step":
        tshape, dshape = PAIRS[case["pair"]]
        spec, draft, rows = model_spec(tshape, case["layers"]), model_spec(dshape, case["draft_layers"]), case["k"] + 1
    else:
        spec, draft, rows = model_spec(case["shape"], case["layers"]), None, case.get("tokens", 1)
    batch = case.get("batch", 1)
    ctx = ragged(case["ctx"], batch) if "ctx" in case else [0]
    pages = -(-(max(ctx) + rows) // 256)
    toks = torch.randint(0, spec.vocab, (batch * (rows if kind == "prefill" else 1),), generator=make_gen(seed, 3), device=DEV).tolist()
    return {"spec": spec, "draft": draft, "batch": batch, "ctx": ctx, "pages": pages, "tokens": toks}


def cached(spec, setup, seed, salt):
    """Keys and values of the contexts, as projections of normed rows leave them: [2, L, pages, 256, KV, hd], zero behind a context."""
    kv = torch.zeros(2, spec.layers, setup["batch"] * setup["pages"], 256, spec.kv_heads, spec.head_dim, dtype=torch.bfloat16, device=DEV)
    rows = kv.view(2, spec.layers, setup["batch"], setup["pages"] * 256, spec.kv_heads, spec.head_dim)
    g = make_gen(seed, salt)
    for b, n in enumerate(setup["ctx"]):
        if n:
            rows[:, :, b, :n] = normal(g, 1.0, 2, spec.layers, n, spec.kv_heads, spec.head_dim)
    return kv


def dense_state(case, seed):
    s = dense_setup(case, seed)
    r = PairRunner(s["spec"], s["draft"], spec_k=case.get("k", 0), max_batch=s["batch"], block_size=256, max_model_len=256 * s["pages"], use_graph=True, use_pdl=True)
    r.bind_weights(L.TARGET, dense_weights(s["spec"], seed, "target"))
    r.kv[L.TARGET].copy_(cached(s["spec"], s, seed, 21))
    if s["draft"]:
        r.bind_weights(L.DRAFT, dense_weights(s["draft"], seed, "draft"))
        r.kv[L.DRAFT].copy_(cached(s["draft"], s, seed, 22))
    r.finalize()
    s["tables"] = [list(range(b * s["pages"], (b + 1) * s["pages"])) for b in range(s["batch"])]
    return {"case": case, "runner": r, **s}


def run_dense(st):
    r, kind, B = st["runner"], st["case"]["kind"], st["batch"]
    if kind == "step":
        toks, accepted, recovery = r.spec_step(st["ctx"], st["tokens"], st["tables"], st["tables"], [0.0] * B, [0.0] * B)
        return {"tokens": toks, "accepted": accepted, "recovery": recovery, "logits_p": r.logits_p(B), "logits_q": r.logits_q(B),
                "kv": r.kv[L.TARGET], "kv_draft": r.kv[L.DRAFT]}
    if kind == "prefill":
        r.prefill(L.TARGET, st["tokens"], st["tables"][0])
    else:
        r.forward_tokens(L.TARGET, [[t] for t in st["tokens"]], st["ctx"], st["tables"])
    return {"logits": r.logits_last(B), "kv": r.kv[L.TARGET]}


# ------------------------------------------------------------------------------------------------ single operations
def op_state(case, seed):
    h, _, H, KV, hd, F, _, eps, theta, _, _ = SHAPES[case["shape"]]
    g = make_gen(seed, 31)
    st = {"case": case, "eps": eps}
    if case["kind"] == "mlp":
        M = case["rows"]
        st.update(x=normal(g, 0.5, M, h), residual=normal(g, 1.0, M, h), norm=1 + normal(g, 0.1, h), gate_up=normal(g, 0.02, 2 * F, h), down=normal(g, 0.01, h, F))
        return st
    B, Q = case["batch"], case["rows"]
    ctx = ragged(case["ctx"], B)
    pages = -(-(max(ctx) + Q) // 256)
    order = torch.randperm(B * pages, generator=g, device=DEV).to(torch.int32).view(B, pages)   # pages as a pool in use hands them out
    pos = torch.cat([torch.arange(n, n + Q, device=DEV) for n in ctx])
    seq = torch.arange(B, device=DEV).repeat_interleave(Q)
    slots = order[seq, pos // 256].long() * 256 + pos % 256
    freq = theta ** (-torch.arange(0, hd, 2, device=DEV, dtype=F64) / hd)
    ang = torch.arange(pages * 256, device=DEV, dtype=F64)[:, None] * freq
    st.update(H=H, KV=KV, hd=hd, Q=Q, qkv=normal(g, 1.0, B * Q, (H + 2 * KV) * hd), table=order.contiguous(), pos=pos, slots=slots.to(torch.int32),
              lens=torch.tensor([n + Q for n in ctx], dtype=torch.int32, device=DEV), rope=torch.cat([ang.cos(), ang.sin()], -1).float().contiguous(),
              k=normal(g, 1.0, B * pages, 256, KV, hd), v=normal(g, 1.0, B * pages, 256, KV, hd), ctx=ctx)
    return st


def run_op(st):
    if st["case"]["kind"] == "mlp":
        y, residual = ops.rms_norm(st["x"], st["norm"], st["eps"], st["residual"])
        return {"out": ops.linear(ops.gate_up_silu(y, st["gate_up"]), st["down"]), "residual": residual}
    H, KV, hd = st["H"], st["KV"], st["hd"]
    q = ops.rope_store_kv(st["qkv"], st["pos"], st["slots"], st["rope"], st["k"], st["v"], H, KV, hd)
    return {"out": ops.paged_attention(q.view(-1, H, hd), st["k"], st["v"], st["table"], st["lens"], st["Q"], hd ** -0.5), "k": st["k"], "v": st["v"]}


# ------------------------------------------------------------------------------------------------ layered models
def hybrid_spec(case):
    z = dict(hybrid_bench.SIZES[case["size"]])
    arch = case["arch"]
    if arch == "kefurax":
        z["layers"] = case["layers"]
        return hybrid_bench.kefurax_spec(z)
    spec = hybrid_bench.lisenex_spec(z) if arch == "lisenex" else hybrid_bench.vegilix_spec(z)
    # one layer: a routed one with a latent cache of its own; differential attention, or the retention
    spec.layers = [spec.layers[{"lisenex": 2, "vegilix": 0, "vegilix_retention": 2}[arch]]]
    return spec


def hybrid_weights(case, spec, seed, device=DEV):
    g = make_gen(seed, 41) if device == DEV else None
    dt = getattr(torch, case["dtype"])
    W = spec.width

    def lin(*shape):
        return (torch.randn(*shape, generator=g, device=device) / shape[-1] ** 0.5).to(dt)

    def vec(mean, std, *shape):
        return (mean + std * torch.randn(*shape, generator=g, device=device)).to(dt)

    def uni(lo, hi, *shape):
        return (lo + (hi - lo) * torch.rand(*shape, generator=g, device=device)).to(dt)

    off = 0.0 if spec.architecture == "Vegilix" else 1.0   # Vegilix keeps its norm weights around zero
    tied = spec.architecture == "Lisenex"
    embed = (torch.randn(spec.vocab, W, generator=g, device=device) / (W ** 0.5 if tied else 1.0)).to(dt)
    w = {"EMBED": embed, "HEAD": embed if tied else lin(spec.vocab, W), "FINAL_NORM": vec(off, 0.1, W), "layers": []}
    for ls in spec.layers:
        H, D, V, G = ls.heads, ls.dim, ls.vdim, ls.kv_heads
        lw = {"NORM": vec(off, 0.1, W)}
        if ls.mixer == "parallel":
            Hd, Gd, Dd, Vd = ls.d_heads, ls.d_kv_heads, ls.d_dim, ls.d_vdim
            Cd = 2 * Gd * Dd + Hd * Vd
            lw.update(PAIR_IN=lin(H * D + G * (D + V) + H * V + Cd + Hd * Vd + 2 * Hd, W), ATTN_OUT=lin(W, H * V), MIX_OUT=lin(W, Hd * Vd), CONV_W=vec(0.0, 0.6, Cd, ls.conv),
                      DELTA_ALOG=uni(-2.0, 0.5, Hd), DELTA_DT_B=uni(-2.0, 1.0, Hd), MIX_NORM=vec(1.0, 0.1, Hd * Vd))
        elif ls.mixer == "mamba1":
            I, N, R = ls.inner, ls.state, ls.dt_rank
            lw.update(SEL_IN=lin(2 * I, W), CONV_W=vec(0.0, 0.5, I, ls.conv), CONV_B=vec(0.0, 0.2, I), SEL_X=lin(R + 2 * N, I), SEL_DT=lin(I, R), SEL_DT_B=uni(-3.0, -0.5, I),
                      SEL_ALOG=uni(-1.2, 1.4, I, N), SEL_D=vec(1.0, 0.2, I), MIX_OUT=lin(W, I))
        elif ls.mixer == "rglru":
            R, nb = ls.inner, ls.blocks
            bs = R // nb
            lw.update(RGLRU_IN=lin(2 * R, W), RGLRU_IN_B=vec(0.0, 0.3, 2 * R), CONV_W=vec(0.0, 0.5, R, ls.conv), CONV_B=vec(0.0, 0.2, R), RGLRU_GATE=lin(nb, 2 * bs, bs),
                      RGLRU_GATE_B=vec(0.0, 0.5, nb, 2 * bs), RGLRU_LAM=uni(-4.0, 0.5, R), MIX_OUT=lin(W, R))
        elif ls.mixer == "latent_attention":
            R, KR = ls.rot_dim, ls.kv_rank
            lw.update(LAT_IN=lin(H * (D + R) + KR + R + H * V, W), LAT_KVNORM=vec(1.0, 0.1, KR), LAT_UV=lin(H * V, KR), LAT_UKT=(lin(H, KR, D).float() * (D / KR) ** 0.5).to(dt).contiguous(), MIX_OUT=lin(W, H * V))
        elif ls.mixer == "attention":
            lw.update(ATTN_IN=lin(2 * (H + G) * D + G * V, W), ATTN_QK_NORM=vec(1.0, 0.1, 2, D), ATTN_DIFF=vec(0.0, 0.1, 4, D), MIX_OUT=lin(W, H * V))
        else:
            lw.update(RET_IN=lin(2 * H * (D + V), W), MIX_OUT=lin(W, H * V))
        lw["NORM2"] = vec(off, 0.1, W)
        if spec.architecture == "Vegilix":
            lw.update(NORM_POST=vec(0.0, 0.1, W), NORM2_POST=vec(0.0, 0.1, W))
        if ls.mlp == "dense":
            lw.update(GLU_IN=lin(2 * ls.ff, W), GLU_OUT=lin(W, ls.ff))
        else:
            lw.update(ROUTER=lin(ls.experts + ls.identity, W), EXPERT_IN=lin(ls.experts, 2 * ls.ff, W), EXPERT_OUT=lin(ls.experts, W, ls.ff), SHARED_IN=lin(2 * ls.shared_ff, W),
                      SHARED_OUT=lin(W, ls.shared_ff))
            if ls.route_bias:
                lw["ROUTER_BIAS"] = vec(0.0, 0.02, ls.experts + ls.identity)
        w["layers"].append(lw)
    return w


def hybrid_tokens(case, vocab, seed):
    """Token ids of every sequence up to the end of the call, and the first position that the call brings."""
    lens = ragged(case["ctx"], case["batch"]) if case["ctx"] else ragged(case["tokens"], case["batch"])
    g = make_gen(seed, 43)
    first = lens if case["ctx"] else [0] * case["batch"]
    return [torch.randint(0, vocab, (n + (1 if case["ctx"] else 0),), generator=g, device=DEV).tolist() for n in lens], first


def hybrid_pages(case):
    return -(-((case["ctx"] or case["tokens"]) + 8) // 64)


def hybrid_state(case, seed):
    spec = hybrid_spec(case)
    seqs, first = hybrid_tokens(case, spec.vocab, seed)
    B, pages = case["batch"], hybrid_pages(case)
    r = HybridRunner(spec, hybrid_weights(case, spec, seed), dtype=case["dtype"], max_tokens=max(16, sum(len(t) for t in seqs) if not case["ctx"] else 2048), max_seqs=B, block_size=64,
                     num_blocks=pages * B, n_slots=B, max_model_len=pages * 64, max_logit_rows=B)
    tables = [list(range(i * pages, (i + 1) * pages)) for i in range(B)]
    for i in range(B):
        if first[i]:
            r.forward([(seqs[i][:first[i]], 0, i, tables[i], [])])
    entries = [(seqs[i][first[i]:], first[i], i, tables[i], [len(seqs[i]) - first[i] - 1]) for i in range(B)]
    return {"case": case, "runner": r, "entries": entries}


def run_hybrid(st):
    r = st["runner"]
    logits, _ = r.forward(st["entries"], temps=[0.0] * len(st["entries"]))
    out = {"logits": logits}
    if r.spec.has_cache:
        out["cache"] = r.cache.view(r.dtype)
    if any(ls.mixer != "latent_attention" for ls in r.spec.layers):
        out["state"] = r.state.view(torch.float32)
    return out


# ------------------------------------------------------------------------------------------------ the interface
def prepare(case, seed):
    if case["kind"] == "hybrid":
        return hybrid_state(case, seed)
    return op_state(case, seed) if case["kind"] in ("mlp", "attention") else dense_state(case, seed)


def run(state):
    kind = state["case"]["kind"]
    if kind == "hybrid":
        return run_hybrid(state)
    return run_op(state) if kind in ("mlp", "attention") else run_dense(state)


def dense_work(spec, rows, head_rows, contexts):
    """One forward: every matrix once, the contexts' keys and values once, logits of the wanted rows."""
    per = spec.hidden * (spec.heads + 2 * spec.kv_heads) * spec.head_dim + spec.hidden * spec.heads * spec.head_dim + 3 * spec.hidden * spec.ffn
    kv = 2 * spec.kv_heads * spec.head_dim
    seen = sum(contexts)
    b = 2 * (spec.layers * (per + kv * (seen + rows)) + spec.vocab * (spec.hidden + head_rows))
    pairs = sum(rows // len(contexts) * (c - (rows // len(contexts) - 1) / 2) for c in contexts)   # (row, visible key) pairs
    f = 2 * spec.layers * (rows * per + 2 * pairs * spec.heads * spec.head_dim) + 2 * head_rows * spec.vocab * spec.hidden
    return b, f


def work(case):
    kind = case["kind"]
    if kind == "hybrid":
        spec = hybrid_spec(case)
        w = hybrid_weights(case, spec, 0, "meta")
        B, es = case["batch"], 2 if case["dtype"] == "bfloat16" else 4
        rows = B if case["ctx"] else sum(ragged(case["tokens"], B))
        ctx = [n + 1 for n in ragged(case["ctx"], B)] if case["ctx"] else ragged(case["tokens"], B)
        b = spec.vocab * spec.width * es + B * spec.vocab * 4 + rows * spec.width * es
        f = 2.0 * B * spec.vocab * spec.width
        for ls, lw in zip(spec.layers, w["layers"]):
            for name, t in lw.items():
                share = min(1.0, rows * ls.top / ls.experts) if name.startswith("EXPERT") else 1.0
                b += t.numel() * es * share
                if t.dim() >= 2 and not name.startswith(("CONV", "SEL_ALOG", "ATTN_DIFF", "ATTN_QK")):
                    f += 2.0 * rows * t.numel() * (ls.top / ls.experts if name.startswith("EXPERT") else 0.5 if name == "LAT_UKT" and not case["ctx"] else 1.0)
            seen = [min(c, ls.window + ls.keep_first) if ls.window else c for c in ctx]
            pairs = sum(seen) if case["ctx"] else sum(s * (c - s / 2) for s, c in zip(seen, ctx))   # (row, visible key) pairs
            if ls.mixer in ("parallel", "attention"):
                b += sum(seen) * ls.kv_heads * (ls.maps * ls.dim + ls.vdim) * es
                f += 2.0 * pairs * ls.heads * ls.maps * (ls.dim + ls.vdim)
            elif ls.mixer == "latent_attention":
                b += sum(seen) * (ls.kv_rank + ls.rot_dim) * es
                f += 2.0 * pairs * ls.heads * (ls.dim + ls.rot_dim + ls.vdim)
            if ls.mixer in ("parallel", "retention"):
                n = ls.d_heads * ls.d_dim * ls.d_vdim if ls.mixer == "parallel" else ls.heads * ls.dim * ls.vdim
                b, f = b + 8.0 * B * n, f + 6.0 * rows * n
            elif ls.mixer == "mamba1":
                b, f = b + 8.0 * B * ls.inner * ls.state, f + 7.0 * rows * ls.inner * ls.state
        return {"bytes": float(b), "flops": float(f)}
    if kind == "mlp":
        h, _, _, _, _, F, *_ = SHAPES[case["shape"]]
        return {"bytes": 2.0 * (3 * h * F + 4 * case["rows"] * h), "flops": 6.0 * case["rows"] * h * F}
    if kind == "attention":
        _, _, H, KV, hd, *_ = SHAPES[case["shape"]]
        B, Q = case["batch"], case["rows"]
        seen = sum(n + Q for n in ragged(case["ctx"], B))
        return {"bytes": 2.0 * (2 * KV * hd * seen + B * Q * (2 * H + 4 * KV) * hd), "flops": 4.0 * Q * seen * H * hd}
    if kind == "step":
        tshape, dshape = PAIRS[case["pair"]]
        B, K, ctx = case["batch"], case["k"], ragged(case["ctx"], case["batch"])
        b, f = dense_work(model_spec(tshape, case["layers"]), B * (K + 1), B * (K + 1), [c + K + 1 for c in ctx])
        for i in range(K + 1):   # the last draft forward only fills the cache
            db, df = dense_work(model_spec(dshape, case["draft_layers"]), B, B if i < K else 0, [c + i + 1 for c in ctx])
            skip = 2 * SHAPES[dshape][0] * SHAPES[dshape][6] if i == K else 0
            b, f = b + db - skip, f + df
        return {"bytes": float(b), "flops": float(f)}
    rows = case["tokens"] if kind == "prefill" else case["batch"]
    ctx = [case["tokens"]] if kind == "prefill" else [c + 1 for c in ragged(case["ctx"], case["batch"])]
    b, f = dense_work(model_spec(case["shape"], case["layers"]), rows, len(ctx), ctx)
    return {"bytes": float(b), "flops": float(f)}


def tolerance(case):
    """About four times what the outputs were measured to be off from exact()."""
    if case.get("dtype") == "float32":   # 2e-6
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"] in ("mlp", "attention"):   # 0.004 and 0.003
        return {"rel": 1.5e-2, "max": 0.3}
    if case["kind"] == "hybrid":   # 0.003 to 0.006
        return {"rel": 2e-2, "max": 0.5}
    return {"rel": 3e-2, "max": 0.5}   # 0.008 to 0.02 by the depth


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def unit(v, eps):
    return v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps)


def silu(z):
    return z * torch.sigmoid(z)


def softplus(z):
    return torch.logaddexp(z, torch.zeros_like(z))


def turn(v, pos, freq, mult=1.0, half=True):
    """v [n, heads, dim] turned by pos * freq in half-apart or adjacent pairs of the first 2 len(freq) entries."""
    ang = pos.to(F64)[:, None, None] * freq
    c, s, m = ang.cos() * mult, ang.sin() * mult, freq.numel()
    out = v.clone()
    ia, ib = (slice(0, m), slice(m, 2 * m)) if half else (slice(0, 2 * m, 2), slice(1, 2 * m, 2))
    a, b = v[..., ia], v[..., ib]
    out[..., ia], out[..., ib] = a * c - b * s, b * c + a * s
    return out


def frequencies(dims, base):
    return base ** (-torch.arange(0, dims, 2, device=DEV, dtype=F64) / dims)


def attend(q, k, v, pos, scale, mask=None, sink=0.0):
    """q [n, H, D] at positions pos over k [c, G, D], v [c, G, V] from position 0: [n, H, V]."""
    H, G = q.shape[1], k.shape[1]
    at = torch.arange(k.shape[0], device=DEV)
    seen = at[None, :] <= pos[:, None]
    if mask:
        seen &= (pos[:, None] - at[None, :] < mask[0]) | (at[None, :] < mask[1])
    out = torch.empty(q.shape[0], H, v.shape[-1], dtype=F64, device=DEV)
    for h in range(H):
        s = ((q[:, h] @ k[:, h * G // H].T) * scale).masked_fill(~seen, -math.inf)
        m = s.max(-1, keepdim=True).values.clamp(min=0.0) if sink else s.max(-1, keepdim=True).values
        e = torch.exp(s - m)
        out[:, h] = (e @ v[:, h * v.shape[1] // H]) / (e.sum(-1, keepdim=True) + sink * torch.exp(-m))
    return out


def dense64(spec, w, kv, tokens, p0):
    """Rows of one sequence from position p0 through a dense decoder; kv [2, L, positions, KV, hd] gets their keys and values."""
    n, H, KV, hd = len(tokens), spec.heads, spec.kv_heads, spec.head_dim
    pos = torch.arange(p0, p0 + n, device=DEV)
    freq = frequencies(hd, spec.rope_theta)
    x = w["embed"][torch.tensor(tokens, device=DEV)].to(F64)
    for i, lw in enumerate(w["layers"]):
        qkv = (unit(x, spec.rms_eps) * lw["input_norm"].to(F64)) @ lw["qkv"].to(F64).T
        q, k, v = (t.reshape(n, -1, hd) for t in qkv.split([H * hd, KV * hd, KV * hd], 1))
        if spec.qk_norm:
            q, k = unit(q, spec.rms_eps) * lw["q_norm"].to(F64), unit(k, spec.rms_eps) * lw["k_norm"].to(F64)
        kv[0, i, p0:p0 + n], kv[1, i, p0:p0 + n] = turn(k, pos, freq), v
        x = x + attend(turn(q, pos, freq), kv[0, i, :p0 + n], kv[1, i, :p0 + n], pos, hd ** -0.5).reshape(n, -1) @ lw["o"].to(F64).T
        gate, up = ((unit(x, spec.rms_eps) * lw["post_norm"].to(F64)) @ lw["gate_up"].to(F64).T).chunk(2, 1)
        x = x + (silu(gate) * up) @ lw["down"].to(F64).T
    return unit(x, spec.rms_eps) * w["final_norm"].to(F64)


def head64(w, rows):
    return torch.cat([rows @ part.to(F64).T for part in w["lm_head"].split(32768)], 1)


def exact_dense(case, seed):
    s = dense_setup(case, seed)
    w = dense_weights(s["spec"], seed, "target")
    kv = cached(s["spec"], s, seed, 21).to(F64)
    by_seq = kv.view(2, s["spec"].layers, s["batch"], -1, *kv.shape[4:])
    if case["kind"] != "step":
        rows = []
        for b, p0 in enumerate(s["ctx"]):
            rows.append(dense64(s["spec"], w, by_seq[:, :, b], s["tokens"] if case["kind"] == "prefill" else [s["tokens"][b]], p0)[-1:])
        return {"logits": head64(w, torch.cat(rows)), "kv": kv}
    K = case["k"]
    wd = dense_weights(s["draft"], seed, "draft")
    kvd = cached(s["draft"], s, seed, 22).to(F64)
    by_seq_d = kvd.view(2, s["draft"].layers, s["batch"], -1, *kvd.shape[4:])
    out = {"tokens": [], "accepted": [], "recovery": [], "logits_p": [], "logits_q": []}
    for b, p0 in enumerate(s["ctx"]):
        toks, lq = [s["tokens"][b]], []
        for i in range(K + 1):
            row = dense64(s["draft"], wd, by_seq_d[:, :, b], toks[-1:], p0 + i)
            if i < K:
                lq.append(head64(wd, row)[0])
                toks.append(int(lq[-1].argmax()))
        lp = head64(w, dense64(s["spec"], w, by_seq[:, :, b], toks, p0))
        best = lp.argmax(-1).tolist()
        n = next((i for i in range(K) if toks[i + 1] != best[i]), K)
        for key, v in (("tokens", toks), ("accepted", n), ("recovery", best[n]), ("logits_p", lp), ("logits_q", torch.stack(lq))):
            out[key].append(v)
    return {"tokens": np.array(out["tokens"]), "accepted": np.array(out["accepted"], np.int32), "recovery": np.array(out["recovery"]),
            "logits_p": torch.stack(out["logits_p"]), "logits_q": torch.stack(out["logits_q"]), "kv": kv, "kv_draft": kvd}


def exact_op(case, seed):
    st = op_state(case, seed)
    if case["kind"] == "mlp":
        r = st["x"].to(F64) + st["residual"].to(F64)
        gate, up = ((unit(r, st["eps"]) * st["norm"].to(F64)) @ st["gate_up"].to(F64).T).chunk(2, 1)
        return {"out": (silu(gate) * up) @ st["down"].to(F64).T, "residual": r}
    H, KV, hd, Q = st["H"], st["KV"], st["hd"], st["Q"]
    freq = frequencies(hd, SHAPES[case["shape"]][8])
    q, k, v = (t.reshape(-1, n, hd).to(F64) for t, n in zip(st["qkv"].split([H * hd, KV * hd, KV * hd], 1), (H, KV, KV)))
    q, k = turn(q, st["pos"], freq), turn(k, st["pos"], freq)
    ck, cv = st["k"].to(F64), st["v"].to(F64)
    ck.view(-1, KV, hd)[st["slots"].long()], cv.view(-1, KV, hd)[st["slots"].long()] = k, v
    out = []
    for b, n in enumerate(st["ctx"]):
        pages, rows = st["table"][b].long(), slice(b * Q, (b + 1) * Q)
        out.append(attend(q[rows], ck[pages].reshape(-1, KV, hd)[:n + Q], cv[pages].reshape(-1, KV, hd)[:n + Q], st["pos"][rows], hd ** -0.5).reshape(Q, -1))
    return {"out": torch.cat(out), "k": ck, "v": cv}


def conv64(u, w, bias=None):
    """Causal convolution over time of every channel: u [n, C], w [C, taps], the last tap on the current row."""
    taps = w.shape[1]
    full = torch.cat([torch.zeros(taps - 1, u.shape[1], dtype=F64, device=DEV), u])
    y = sum(full[j:j + u.shape[0]] * w[:, j] for j in range(taps))
    return y if bias is None else y + bias


def yarn(ls):
    f = frequencies(ls.rot_dims, ls.rot_base).tolist()

    def dim_of(turns):
        return ls.rot_dims * math.log(ls.yarn_original / (2.0 * math.pi * turns)) / (2.0 * math.log(ls.rot_base))

    lo, hi = max(math.floor(dim_of(ls.yarn_fast)), 0), min(math.ceil(dim_of(ls.yarn_slow)), ls.rot_dims - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(len(f))]
    return torch.tensor([x / ls.yarn_factor * r + x * (1.0 - r) for x, r in zip(f, ramp)], dtype=F64, device=DEV), 0.1 * math.log(ls.yarn_factor) + 1.0


def waves(ls):
    out = []
    for f in frequencies(ls.rot_dims, ls.rot_base).tolist():
        t = ls.wave_original * f / (2.0 * math.pi)
        s = min(max((t - ls.wave_low) / (ls.wave_high - ls.wave_low), 0.0), 1.0)
        out.append((1.0 - s) * f / ls.wave_factor + s * f)
    return torch.tensor(out, dtype=F64, device=DEV)


def mixer64(ls, w, h, eps):
    """One whole sequence from position 0: (result rows, the rows that the cache keeps or None)."""
    n, H, D, V, G = h.shape[0], ls.heads, ls.dim, ls.vdim, ls.kv_heads
    pos = torch.arange(n, device=DEV)
    if ls.mixer == "parallel":
        Hd, Gd, Dd, Vd = ls.d_heads, ls.d_kv_heads, ls.d_dim, ls.d_vdim
        q, k, v, gate, dq, dk, dv, dg, beta, a = (h @ w["PAIR_IN"].T).split([H * D, G * D, G * V, H * V, Gd * Dd, Gd * Dd, Hd * Vd, Hd * Vd, Hd, Hd], 1)
        freq, mult = yarn(ls)
        q, k = (unit(turn(t.reshape(n, -1, D), pos, freq, mult, half=False), eps) for t in (q, k))
        left = attend(q, k, v.reshape(n, G, V), pos, ls.attn_scale, sink=ls.sink).reshape(n, -1) * torch.sigmoid(gate)
        dq, dk, dv = (silu(t) for t in conv64(torch.cat([dq, dk, dv], 1), w["CONV_W"]).split([Gd * Dd, Gd * Dd, Hd * Vd], 1))
        dq, dk, dv = (t.reshape(n, -1, d).repeat_interleave(Hd // g, 1) for t, d, g in ((dq, Dd, Gd), (dk, Dd, Gd), (dv, Vd, Hd)))
        dq, dk = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (dq, dk))
        beta, decay = torch.sigmoid(beta), torch.exp(-torch.exp(w["DELTA_ALOG"]) * softplus(a + w["DELTA_DT_B"]))
        S, o = torch.zeros(Hd, Dd, Vd, dtype=F64, device=DEV), torch.empty(n, Hd, Vd, dtype=F64, device=DEV)
        for t in range(n):
            S = decay[t][:, None, None] * S
            u = beta[t][:, None] * (dv[t] - (dk[t][:, None] @ S)[:, 0])
            S = torch.baddbmm(S, dk[t][:, :, None], u[:, None])
            o[t] = (dq[t][:, None] @ S)[:, 0]
        right = (unit(o * Dd ** -0.5, eps).reshape(n, -1) * w["MIX_NORM"]) * silu(dg)
        return ls.left_scale * left @ w["ATTN_OUT"].T + ls.right_scale * right @ w["MIX_OUT"].T, torch.cat([k.reshape(n, -1), v], 1)
    if ls.mixer == "mamba1":
        x, z = (h @ w["SEL_IN"].T).chunk(2, 1)
        x = silu(conv64(x, w["CONV_W"], w["CONV_B"]))
        dt, Bm, Cm = (x @ w["SEL_X"].T).split([ls.dt_rank, ls.state, ls.state], 1)
        dt = softplus(dt @ w["SEL_DT"].T + w["SEL_DT_B"])
        A, S, y = -torch.exp(w["SEL_ALOG"]), torch.zeros(ls.inner, ls.state, dtype=F64, device=DEV), torch.empty_like(x)
        for t in range(n):
            S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * x[t])[:, None] * Bm[t]
            y[t] = S @ Cm[t]
        return ((y + w["SEL_D"] * x) * silu(z)) @ w["MIX_OUT"].T, None
    if ls.mixer == "rglru":
        R, nb = ls.inner, ls.blocks
        y, u = (h @ w["RGLRU_IN"].T + w["RGLRU_IN_B"]).chunk(2, 1)
        u = conv64(u, w["CONV_W"], w["CONV_B"])
        r, i = torch.sigmoid(torch.einsum("nbi,boi->nbo", u.reshape(n, nb, -1), w["RGLRU_GATE"]) + w["RGLRU_GATE_B"]).chunk(2, 2)
        a = torch.exp(-ls.decay_mult * r.reshape(n, R) * softplus(w["RGLRU_LAM"]))
        inp, S, o = torch.sqrt(1.0 - a * a) * i.reshape(n, R) * u, torch.zeros(R, dtype=F64, device=DEV), torch.empty_like(u)
        for t in range(n):
            S = o[t] = a[t] * S + inp[t]
        return (o * torch.nn.functional.gelu(y, approximate="tanh")) @ w["MIX_OUT"].T, None
    if ls.mixer == "latent_attention":
        R, KR = ls.rot_dim, ls.kv_rank
        q, lat, kr, gate = (h @ w["LAT_IN"].T).split([H * (D + R), KR, R, H * V], 1)
        freq = frequencies(ls.rot_dims, ls.rot_base)
        lat, kr, q = unit(lat, eps) * w["LAT_KVNORM"], turn(kr.reshape(n, 1, R), pos, freq, half=False), q.reshape(n, H, D + R)
        q = torch.cat([q[..., :D], turn(q[..., D:], pos, freq, half=False)], -1)
        k = torch.cat([torch.einsum("nk,hkd->nhd", lat, w["LAT_UKT"]), kr.expand(n, H, R)], -1)
        o = attend(q, k, (lat @ w["LAT_UV"].T).reshape(n, H, V), pos, ls.attn_scale).reshape(n, -1)
        return (o * torch.sigmoid(gate)) @ w["MIX_OUT"].T, torch.cat([lat, kr[:, 0]], 1)
    if ls.mixer == "attention":
        q, k, v = (h @ w["ATTN_IN"].T).split([2 * H * D, 2 * G * D, G * V], 1)
        freq = waves(ls)
        q, k = (turn(unit(t.reshape(n, -1, D), eps) * w["ATTN_QK_NORM"][j], pos, freq) for j, t in enumerate((q, k)))
        lq1, lk1, lq2, lk2 = w["ATTN_DIFF"]
        lam = torch.exp((lq1 * lk1).sum()) - torch.exp((lq2 * lk2).sum()) + ls.diff
        a1, a2 = (attend(q[:, j::2], k[:, j::2], v.reshape(n, G, V), pos, ls.attn_scale, (ls.window, ls.keep_first)) for j in (0, 1))
        return (unit(a1 - lam * a2, eps) * (1.0 - ls.diff)).reshape(n, -1) @ w["MIX_OUT"].T, torch.cat([k.reshape(n, -1), v], 1)
    q, k, v, gate = (h @ w["RET_IN"].T).split([H * D, H * D, H * V, H * V], 1)
    freq = frequencies(ls.rot_dims, ls.rot_base)
    q, k, v = turn(q.reshape(n, H, D), pos, freq), turn(k.reshape(n, H, D), pos, freq) * D ** -0.5, v.reshape(n, H, V)
    o = torch.empty(n, H, V, dtype=F64, device=DEV)
    back = pos[:, None] - pos[None, :]
    for j, d in enumerate(ls.decay):
        o[:, j] = ((q[:, j] @ k[:, j].T) * torch.where(back >= 0, d ** back.clamp(min=0).to(F64), 0.0)) @ v[:, j]
    return (unit(o, eps).reshape(n, -1) * silu(gate)) @ w["MIX_OUT"].T, None


def ff64(ls, w, h):
    def glu(rows, up, down, act):
        g, u = (rows @ up.to(F64).T).chunk(2, 1)
        return (act(g) * u) @ down.to(F64).T

    if ls.mlp == "dense":
        return glu(h, w["GLU_IN"], w["GLU_OUT"], lambda z: torch.nn.functional.gelu(z, approximate="tanh"))
    z = h @ w["ROUTER"].T
    if ls.route_softmax:
        score = torch.softmax(z, -1)
        choice = score + w["ROUTER_BIAS"]
        best = choice.reshape(-1, ls.groups, z.shape[1] // ls.groups).max(-1).values.topk(ls.keep, -1).indices
        kept = torch.zeros(z.shape[0], ls.groups, dtype=torch.bool, device=DEV).scatter(1, best, True).repeat_interleave(z.shape[1] // ls.groups, 1)
        sel = choice.masked_fill(~kept, -math.inf).topk(ls.top, -1).indices
        wts = score.gather(1, sel) * ls.route_scale
    else:
        sel = z.topk(ls.top, -1).indices
        wts = torch.softmax(z.gather(1, sel), -1) * ls.route_scale
    out = glu(h, w["SHARED_IN"], w["SHARED_OUT"], silu)
    for j in range(ls.experts + ls.identity):
        row, place = (sel == j).nonzero(as_tuple=True)
        if row.numel():
            y = h[row] if j >= ls.experts else glu(h[row], w["EXPERT_IN"][j], w["EXPERT_OUT"][j], silu)
            out.index_add_(0, row, y * wts[row, place][:, None])
    return out


def exact_hybrid(case, seed):
    spec = hybrid_spec(case)
    raw = hybrid_weights(case, spec, seed)
    seqs, _ = hybrid_tokens(case, spec.vocab, seed)
    layers = [{k: t if k.startswith("EXPERT") else t.to(F64) for k, t in lw.items()} for lw in raw["layers"]]
    eps, mult, rows = spec.eps, spec.residual_mult, []
    pools = [None] * len(layers)
    for b, toks in enumerate(seqs):
        x = raw["EMBED"][torch.tensor(toks, device=DEV)].to(F64) * spec.embed_scale
        for i, (ls, w) in enumerate(zip(spec.layers, layers)):
            if spec.architecture == "Kefurax":
                y, keep = mixer64(ls, w, x, eps)
                x = x + mult * unit(y, eps) * w["NORM"]
                x = x + mult * unit(ff64(ls, w, x), eps) * w["NORM2"]
            elif spec.architecture == "Lisenex":
                y, keep = mixer64(ls, w, unit(x, eps) * w["NORM"], eps)
                x = x + y + ff64(ls, w, unit(x, eps) * w["NORM2"])
            else:
                y, keep = mixer64(ls, w, unit(x, eps) * (1.0 + w["NORM"]), eps)
                x = x + mult * unit(y, eps) * (1.0 + w["NORM_POST"])
                x = x + mult * unit(ff64(ls, w, unit(x, eps) * (1.0 + w["NORM2"])), eps) * (1.0 + w["NORM2_POST"])
            if keep is not None:
                if pools[i] is None:
                    pools[i] = torch.zeros(case["batch"], hybrid_pages(case) * 64, keep.shape[1], dtype=F64, device=DEV)
                pools[i][b, :keep.shape[0]] = keep
        norm = raw["FINAL_NORM"].to(F64) + (1.0 if spec.architecture == "Vegilix" else 0.0)
        rows.append(unit(x[-1:], eps) * norm)
    out = {"logits": torch.cat(rows) @ raw["HEAD"].to(F64).T}
    if any(p is not None for p in pools):
        out["cache"] = torch.cat([p.reshape(-1) for p in pools if p is not None])
    if any(ls.mixer != "latent_attention" for ls in spec.layers):
        out["state"] = None   # kept in a layout of the implementation's own
    return out


def exact(case, seed):
    if case["kind"] == "hybrid":
        return exact_hybrid(case, seed)
    return exact_op(case, seed) if case["kind"] in ("mlp", "attention") else exact_dense(case, seed)
