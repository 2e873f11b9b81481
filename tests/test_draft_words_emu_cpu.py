"""csrc/draft_stream.cuh on host threads with the exchange of the product (tagged words that their readers poll; tests/test_draft_stream_emu_cpu.py runs the
same source with barriers in their place, and only that form), for one sequence and for batches of uneven contexts: logits of every forward, keys and values, tokens (greedy and Philox)
against the oracle, two launches over the same words.  What it cannot show is the device's memory model and speed."""
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

from oracle.model import ModelCfg, OracleModel, random_weights

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "emu", "run_draft_words.cpp")
BIN = os.path.join(ROOT, "tests", "emu", "_build", "run_draft_words")
ASAN = BIN + "_asan"   # every access outside an array of the runner ends the process
# SSD_B200_TSAN=1: the words' runner with ThreadSanitizer, which reports what two threads touch without an order between them (the words are atomic, and a value travels in its word)
TSAN = os.environ.get("SSD_B200_TSAN") == "1"
if TSAN:
    BIN += "_tsan"

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++ (C++20)")


def _build(binary=BIN):
    flags = ["-fsanitize=address", "-g"] if binary == ASAN else (["-fsanitize=thread", "-g"] if TSAN else [])
    deps = [SRC, os.path.join(ROOT, "tests", "emu", "cuda_emu.h")] + [os.path.join(ROOT, "ssd_b200", "csrc", n) for n in ("draft_stream.cuh", "common.cuh", "sampling.cuh")]
    if os.path.exists(binary) and all(os.path.getmtime(binary) >= os.path.getmtime(d) for d in deps):
        return
    os.makedirs(os.path.dirname(binary), exist_ok=True)
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", "-Wno-unknown-pragmas", "-Wno-attributes", *flags, "-o", binary, SRC], check=True)


def _u16(t):
    return t.contiguous().view(torch.int16).numpy().astype(np.uint16)


def _check(tmp_path, hd, kv, grid, ffn, ctx, temp, chunk, bs=16, unnamed=(), binary=BIN, lose=()):
    """One launch against the oracle.  unnamed: (sequence, entry) pairs of the page tables that name no page."""
    from oracle import verify as V
    _build(binary)
    torch.manual_seed(3)
    B, n_fwd = len(ctx), 2
    cfg = ModelCfg(hidden=256, layers=1 if ffn > 4096 else 2, heads=256 // hd, kv_heads=kv, head_dim=hd, ffn=ffn, vocab=264, max_pos=1024, rms_eps=1e-6, rope_theta=500000.0, qk_norm=hd == 128)
    w = random_weights(cfg, seed=9)
    per = (max(ctx) + n_fwd) // bs + 1
    nblk = B * per
    order = torch.randperm(nblk).tolist()
    tables = [order[b * per:(b + 1) * per] for b in range(B)]
    model = OracleModel(cfg, w, num_blocks=nblk, block_size=bs)
    given = [[-1 if (b, i) in unnamed else t for i, t in enumerate(row)] for b, row in enumerate(tables)]
    for b, n in enumerate(ctx):
        if not n:
            continue
        slots = torch.tensor([tables[b][p // bs] * bs + p % bs for p in range(n)], dtype=torch.int32)
        model.forward(torch.randint(0, cfg.vocab, (n,)), torch.arange(n), slots, torch.tensor([n], dtype=torch.int32), torch.tensor([tables[b]], dtype=torch.int32), n)
    for b, i in unnamed:   # tokens without a page: keys and values of zeros, and nothing is stored (the oracle reads a page of zeros that the kernel does not know)
        model.kv_cache[:, :, tables[b][i]] = 0
    kv0 = model.kv_cache.clone()
    for b, i in unnamed:
        kv0[:, :, tables[b][i]] = 3.0
    seed, call_base = 1234, 7 * 16
    temps = [temp if b != 1 else 0.0 for b in range(B)]
    blob, out = tmp_path / "in.bin", tmp_path / "out.bin"
    with open(blob, "wb") as f:
        np.array([B, cfg.hidden, cfg.layers, cfg.heads, cfg.kv_heads, hd, cfg.ffn, cfg.vocab, int(cfg.qk_norm), bs, per, nblk * bs, n_fwd, grid, cfg.max_pos, 4, chunk], dtype=np.int32).tofile(f)
        np.array([cfg.rms_eps] + temps, dtype=np.float32).tofile(f)
        np.array([seed, call_base], dtype=np.uint64).tofile(f)
        np.array([77 + b for b in range(B)], dtype=np.int64).tofile(f)
        np.array(ctx, dtype=np.int32).tofile(f)
        np.array(given, dtype=np.int32).tofile(f)
        for t in (w["embed"], w["final_norm"], w["lm_head"]):
            _u16(t).tofile(f)
        model.rope.numpy().astype(np.float32).tofile(f)
        ones = torch.ones(hd, dtype=torch.bfloat16)
        for lw in w["layers"]:
            for k in ("qkv", "o", "gate_up", "down", "input_norm", "post_norm"):
                _u16(lw[k]).tofile(f)
            _u16(lw.get("q_norm", ones)).tofile(f)
            _u16(lw.get("k_norm", ones)).tofile(f)
        _u16(kv0[0]).tofile(f)
        _u16(kv0[1]).tofile(f)
    res = subprocess.run([binary, str(blob), str(out), *lose], capture_output=True, text=True, timeout=600)
    assert res.returncode == 0, res.stderr[-2000:]
    assert "ThreadSanitizer" not in res.stderr, res.stderr[:3000]
    raw = np.fromfile(out, dtype=np.uint16)
    nl, nc = B * n_fwd * cfg.vocab, cfg.layers * nblk * bs * kv * hd
    bf = torch.from_numpy(raw[:nl + 2 * nc].astype(np.int16)).view(torch.bfloat16)
    logits, kc, vc = bf[:nl].reshape(B, n_fwd, cfg.vocab), bf[nl:nl + nc].float(), bf[nl + nc:].float()
    toks = np.frombuffer(raw[nl + 2 * nc:].tobytes(), dtype=np.int64).reshape(B, n_fwd + 1)
    for b, n in enumerate(ctx):
        bt = torch.tensor([tables[b]], dtype=torch.int32)
        for step in range(n_fwd):
            p = n + step
            slot = torch.tensor([given[b][p // bs] * bs + p % bs if given[b][p // bs] >= 0 else -1], dtype=torch.int32)
            h = model.forward(torch.tensor([int(toks[b, step])]), torch.tensor([p]), slot, torch.tensor([p + 1], dtype=torch.int32), bt, 1)
            if step == n_fwd - 1:
                assert toks[b, step + 1] == -1   # the last forward has no head
                break
            want, got = model.compute_logits(h)[0].float(), logits[b, step].float()
            # bf16 roundings of the hidden state (2^-9 each, about sixteen of them on the way) on logits of unit scale
            assert (got - want).abs().max() <= 0.02 * want.abs().max() + 0.02, (b, step)
            # the token is what the sampler's rule makes of the kernel's own logits
            row = logits[:, step] if temps[b] else logits[b, step][None]
            mine = V.sample(row, torch.tensor(temps if temps[b] else [0.0]), seed, call_base + step)
            assert toks[b, step + 1] == int(mine[b if temps[b] else 0]), (b, step)
    for b, i in unnamed:
        model.kv_cache[:, :, tables[b][i]] = 3.0   # (untouched)
    ref = model.kv_cache.float()
    for got, want in ((kc, ref[0].reshape(-1)), (vc, ref[1].reshape(-1))):
        assert (got - want).abs().max() <= 0.02 * want.abs().max() + 1e-3


@pytest.mark.parametrize("hd,kv,grid,ffn,ctx,temp,chunk", [
    (64, 2, 3, 512, [21], 0.0, 1024),                # one sequence, a range per key head
    (64, 1, 2, 512, [300], 0.7, 256),                # two ranges: exchange of partial results; two slots per tile
    (128, 1, 3, 768, [270, 5, 33], 0.0, 256),        # three sequences on the instance of four, three slots per tile
    (64, 2, 2, 512, [9, 255, 256, 1, 30], 0.8, 512), # five: fragments straight from the words; more units than CTAs, contexts around a round of keys
    (64, 1, 2, 512, [600], 0.0, 512),                # a table of 38 pages, which stays in global memory; ranges of 320 keys, two rounds
    (64, 1, 2, 5120, [21], 0.7, 2048),               # an intermediate row of four slots of five steps
    (64, 1, 2, 4608, [40, 3, 7], 0.0, 2048),         # an intermediate row too long for the shared memory of four tokens' instance
])
def test_tagged_exchange_matches_the_oracle(tmp_path, hd, kv, grid, ffn, ctx, temp, chunk):
    _check(tmp_path, hd, kv, grid, ffn, ctx, temp, chunk)


@pytest.mark.parametrize("hd,ctx,bs,unnamed", [
    (64, [0], 16, [(0, 0)]),                           # no token in the cache and no page for the first
    (128, [0, 30], 32, [(0, 0)]),                      # the same beside a sequence that has pages, pages of whole 32 keys
    (64, [15, 40], 16, [(0, 0), (1, 1)]),              # a first page, whose last slot the new token would take; one inside a context
    (64, [70, 40], 32, [(0, 1), (0, 2), (1, 1)]),      # pages of whole 32 keys, among them the new token's
])
def test_tokens_without_a_page_are_zeros(tmp_path, hd, ctx, bs, unnamed):
    """The rule of paged_attn_kernel, and no read outside the cache (address sanitizer)."""
    _check(tmp_path, hd, 2 if hd == 64 else 1, 2, 512, ctx, 0.0, 512, bs=bs, unnamed=unnamed, binary=ASAN)


def test_attention_weights_keep_all_their_bits():
    """The products take a weight as bf16 pieces; their sum is the 32-bit weight."""
    _build()
    res = subprocess.run([BIN, "pieces"], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stderr[-500:]


@pytest.mark.parametrize("lose", [("words", "0"), ("words", "700"), ("copies", "0"), ("copies", "60"), ("copies", "900")])
def test_waits_that_run_out_end_the_launch(tmp_path, lose):
    """What the last CTA sends, or the weights that it fetches, is lost on the way: every wait for it has a limit, the launch ends with its word set, and the next one is right (the
    runner looks at the word, the barrier's count and the range of the tokens behind both)."""
    _check(tmp_path, 64, 1, 2, 512, [40, 300], 0.7, 256, lose=lose)


def test_register_split_fits_the_launch():
    """Eight consumer warps of 232 registers and four warps of 40 come out of what twelve warps are launched with: fewer would wait for ever, and a build with another number turns the
    form off (it may have more, up to what the split leaves a consumer)."""
    _build()
    res = subprocess.run([BIN, "registers"], capture_output=True, text=True, timeout=60)
    assert [int(x) for x in res.stdout.split()] == list(range((8 * 232 + 4 * 40 + 11) // 12, 233))
