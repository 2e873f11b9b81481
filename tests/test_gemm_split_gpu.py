"""fp32 products as three bf16 pieces on the tensor cores (gemm_split_kernel) against the float64 oracles, forced on for every product that
it can take, and beside the FMA form: prompts around its tile edges, portions, single tokens, grouped experts, batched heads."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# A product of 2^-24 terms summed over k <= 600 and a handful of products in a row stay below 1e-6 .. 1e-5; a piece left out shows as 2^-16.
TOL = 2e-5


def _model(arch):
    U = importlib.import_module(f"tests.{arch}_util")
    if arch == "vegilix":
        cfg = U.config([U.attention(heads=4, kv_heads=2, dim=16, vdim=24, dims=8, window=40, mlp=U.moe(experts=5, top=2, ff=48, shared_ff=16)),
                        U.retention(heads=2, dim=16, vdim=8, dims=8)], width=600, vocab=64)
        plain = importlib.import_module("tests.vegilix_plain").PlainModel
    else:
        cfg = U.config([U.parallel(left=U.attention(heads=4, kv_heads=2, dim=16, vdim=8, dims=8), right=U.delta(heads=4, kv_heads=2, dim=16, vdim=8), mlp=U.dense(320)),
                        U.rglru(width=48, blocks=2), U.mamba1(inner=64, state=8, dt_rank=8)], width=264, vocab=72)
        plain = U.PlainModel
    return U, cfg, plain


@pytest.mark.parametrize("arch", ["vegilix", "kefurax"])
def test_three_pieces_match_the_oracle(tmp_path, monkeypatch, arch):
    from ssd_b200.hybrid import HybridRunner, HybridSpec, load_hybrid_weights
    U, cfg, plain_type = _model(arch)
    tensors = U.random_tensors(cfg, 1)
    path = U.write_checkpoint(str(tmp_path / "ckpt"), cfg, tensors)
    spec = HybridSpec.from_dir(path)
    w = load_hybrid_weights(path, spec, torch.float32, "cuda:0")
    plain = plain_type(cfg, tensors)
    runners = {}
    for mode in ("0", "2"):
        monkeypatch.setenv("SSDK_HYB_SPLIT", mode)
        runners[mode] = HybridRunner(spec, w, dtype="float32", max_tokens=300, max_seqs=2, block_size=16, num_blocks=40, n_slots=2, max_model_len=320)
    toks = torch.randint(0, cfg["vocab"], (261,), generator=torch.Generator().manual_seed(2)).tolist()
    want = plain.run(toks).numpy()
    pages = list(range(20))
    for cuts in ([261], [128, 129, 1, 1, 2], [31, 33, 65, 127, 5]):
        errs = {}
        for mode, r in runners.items():
            got, at = [], 0
            for n in cuts:
                got.append(r.forward([(toks[at:at + n], at, 1, pages, list(range(n)))])[0])
                at += n
            errs[mode] = U.rel_err(np.concatenate(got), want)
        assert errs["2"] < TOL and errs["2"] < max(1e-6, 1.5 * errs["0"]), (cuts, errs)


def test_infinite_largest_and_tiny_operands(tmp_path, monkeypatch):
    """Operands that three bf16 pieces cannot hold give what the FMA form gives: the same infinities and NaNs, the same numbers for values
    above bf16's largest and for results of any size.  Wide head rows (whole products), few and many rows, split k, and one expert."""
    from ssd_b200.hybrid import HybridRunner, HybridSpec, load_hybrid_weights
    U, cfg, _ = _model("vegilix")
    path = U.write_checkpoint(str(tmp_path / "ckpt"), cfg, U.random_tensors(cfg, 1))
    spec = HybridSpec.from_dir(path)
    inf, big, g = float("inf"), 3.395e38, torch.Generator().manual_seed(4)
    small = [1e-20, 1e-27, 1e-33, 1e-36]

    def run(mode, change):
        monkeypatch.setenv("SSDK_HYB_SPLIT", mode)
        w = load_hybrid_weights(path, spec, torch.float32, "cuda:0")
        change(w)
        r = HybridRunner(spec, w, dtype="float32", max_tokens=300, max_seqs=2, block_size=16, num_blocks=40, n_slots=2, max_model_len=320)
        toks = torch.randint(0, cfg["vocab"], (261,), generator=torch.Generator().manual_seed(2)).tolist()
        out = [r.forward([(toks[:n], 0, 0, list(range(20)), list(range(n)))])[0] for n in (1, 7, 261)]
        r.close()
        return np.concatenate(out)

    def head(w):
        h = w["HEAD"]
        h[3, 7] = inf
        h[5, 0], h[5, 599] = inf, -inf
        h[9, 64] = big
        h[10] = h[10] * 1e-3
        h[10, 300] = -big
        h[11, 1] = float("nan")
        for i, f in enumerate(small):
            h[20 + i] = h[20 + i] * f

    def expert(w):
        w["layers"][0]["EXPERT_IN"].view(-1, 600)[17, 5] = inf

    with np.errstate(all="ignore"):
        for change in (head, expert):
            a, b = run("0", change), run("2", change)
            assert not np.isfinite(a).all()
            assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(np.where(np.isinf(a), np.sign(a), 0), np.where(np.isinf(b), np.sign(b), 0))
        a, b = (run(mode, head).astype(np.float64) for mode in ("0", "2"))
    for col in [9, 10, 20, 21, 22, 23]:
        ok = np.isfinite(a[:, col])
        x, y = a[ok, col], b[ok, col]
        size = np.abs(x).max()   # (the squares of 1e-36 are not numbers)
        assert ok.any() and np.linalg.norm((x - y) / size) < TOL * np.linalg.norm(x / size), col


def test_many_tiles_per_pair(tmp_path, monkeypatch):
    """1000 rows through a head of 8000 columns and k = 328: 256 tiles, three and four per pair of CTAs on 148 SMs, so that rings and
    accumulators run on from tile to tile; against the float64 oracle."""
    from ssd_b200.hybrid import HybridRunner, HybridSpec, load_hybrid_weights
    U = importlib.import_module("tests.kefurax_util")
    cfg = U.config([U.rglru(width=48, blocks=2)], width=328, vocab=8000)
    tensors = U.random_tensors(cfg, 6)
    path = U.write_checkpoint(str(tmp_path / "ckpt"), cfg, tensors)
    spec = HybridSpec.from_dir(path)
    w = load_hybrid_weights(path, spec, torch.float32, "cuda:0")
    toks = torch.randint(0, cfg["vocab"], (1000,), generator=torch.Generator().manual_seed(2)).tolist()
    want = U.PlainModel(cfg, tensors).run(toks).numpy()
    errs = {}
    for mode in ("0", "2"):
        monkeypatch.setenv("SSDK_HYB_SPLIT", mode)
        r = HybridRunner(spec, w, dtype="float32", max_tokens=1000, max_seqs=1, block_size=16, num_blocks=64, n_slots=1, max_model_len=1024)
        got = r.forward([(toks, 0, 0, list(range(63)), list(range(1000)))])[0]
        errs[mode] = np.sqrt(((got - want) ** 2).mean(-1) / (want ** 2).mean(-1)).max()   # the worst row
        r.close()
    assert errs["2"] < TOL and errs["2"] < max(1e-6, 1.5 * errs["0"]), errs


def test_many_expert_tiles(tmp_path, monkeypatch):
    """40 experts of 520 columns over 1000 rows: 200 grouped tiles of 5 to 100 rows, against the FMA form (its error is 1e-6)."""
    from ssd_b200.hybrid import HybridRunner, HybridSpec, load_hybrid_weights
    U = importlib.import_module("tests.vegilix_util")
    cfg = U.config([U.retention(heads=2, dim=16, vdim=8, dims=8, mlp=U.moe(experts=40, top=2, ff=520, shared_ff=16))], width=600, vocab=64)
    path = U.write_checkpoint(str(tmp_path / "ckpt"), cfg, U.random_tensors(cfg, 1))
    spec = HybridSpec.from_dir(path)
    w = load_hybrid_weights(path, spec, torch.float32, "cuda:0")
    toks = torch.randint(0, cfg["vocab"], (1000,), generator=torch.Generator().manual_seed(2)).tolist()
    out = []
    for mode in ("0", "2"):
        monkeypatch.setenv("SSDK_HYB_SPLIT", mode)
        r = HybridRunner(spec, w, dtype="float32", max_tokens=1000, max_seqs=1, block_size=16, num_blocks=64, n_slots=1, max_model_len=1024)
        out.append(r.forward([(toks, 0, 0, list(range(63)), list(range(1000)))])[0].copy())
        r.close()
    err = np.sqrt(((out[0] - out[1]) ** 2).mean(-1) / (out[0] ** 2).mean(-1))
    assert np.isfinite(out[1]).all() and err.max() < TOL, f"row {err.argmax()} off by {err.max():.2e}"
