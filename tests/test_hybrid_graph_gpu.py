"""Decode steps replayed as graphs, and programmatic dependent launch, give the bits of plain launches: every design, contexts that cross
the attention's split edges, greedy and sampled rows, changed batches, and steps without logits or tokens in between."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(spec, w, dtype, monkeypatch, plain):
    from ssd_b200.hybrid import HybridRunner
    monkeypatch.setenv("SSDK_HYB_GRAPH", "0" if plain else "1")
    monkeypatch.setenv("SSDK_HYB_PDL", "0" if plain else "1")
    r = HybridRunner(spec, w, dtype=dtype, max_tokens=256, max_seqs=3, block_size=16, num_blocks=48, n_slots=3, max_model_len=256)
    g = torch.Generator().manual_seed(1)
    tables = [list(range(16 * i, 16 * (i + 1))) for i in range(3)]
    pos = [121, 63, 7]
    out = [r.forward([(torch.randint(0, spec.vocab, (pos[i],), generator=g).tolist(), 0, i, tables[i], [pos[i] - 1]) for i in range(3)])[0]]
    toks = torch.randint(0, spec.vocab, (3,), generator=g).tolist()
    for step in range(14):
        live = [0, 1, 2] if step % 5 else [2, 0]
        temps = [0.0, 0.8, 0.0][:len(live)] if step % 4 != 3 else None
        lg, tk = r.forward([([toks[i]], pos[i], i, tables[i], [0]) for i in live], temps=temps, seed=11)
        out.append(lg)
        for j, i in enumerate(live):
            pos[i] += 1
            toks[i] = tk[j] if tk is not None else int(lg[j].argmax())
        out.append(np.array([toks]))
    count = r.launch_count
    r.close()
    return out, count


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("arch", ["pikavik", "kefurax", "lisenex", "kokatar", "vatolorn", "vegilix"])
def test_same_bits_as_plain_launches(monkeypatch, arch, dtype):
    from ssd_b200 import hybrid_bench as hb
    from ssd_b200.hybrid import random_hybrid_weights
    spec = getattr(hb, arch + "_spec")(dict(hb.SIZES["s"], layers=4, vocab=1000))
    w = random_hybrid_weights(spec, getattr(torch, dtype), "cuda:0", seed=2)
    want, n_plain = _run(spec, w, dtype, monkeypatch, True)
    got, n = _run(spec, w, dtype, monkeypatch, False)
    assert n == n_plain
    for i, (a, b) in enumerate(zip(want, got)):
        assert np.array_equal(a, b), f"output {i}"


def _decode(r, n, pos, sample):
    temps = [0.0] * n if sample else None
    return r.forward([([7 + i], pos, i, [i], [0]) for i in range(n)], temps=temps)


def test_kinds_of_steps_keep_their_graphs(monkeypatch):
    """A kind of step gets its graph once: not again while other kinds come and go (more of them than are kept), nor along a context whose
    splits stay; kinds that come up a few times get none.  The numbers are those of plain launches throughout."""
    from ssd_b200 import hybrid_bench as hb
    from ssd_b200.hybrid import HybridRunner, random_hybrid_weights
    spec = hb.kokatar_spec(dict(hb.SIZES["s"], layers=1, vocab=512))
    w = random_hybrid_weights(spec, torch.bfloat16, "cuda:0", seed=2)
    runners = []
    for plain in (True, False):
        monkeypatch.setenv("SSDK_HYB_GRAPH", "0" if plain else "1")
        runners.append(HybridRunner(spec, w, max_tokens=64, max_seqs=40, block_size=1024, num_blocks=40, n_slots=40, max_model_len=1024))
    made = lambda: runners[1].lib.ssdk_hyb_graphs_made(runners[1].h)

    def both(*a):
        (la, ta), (lb, tb) = (_decode(r, *a) for r in runners)
        assert np.array_equal(la, lb) and ta == tb

    for _ in range(3):
        both(3, 5, True)
    assert made() == 0
    for n in (1, 2, 3):
        for _ in range(8):
            both(n, 5, True)
    assert made() == 3
    for n in range(4, 41):   # 74 other kinds, each of them twice, the first three in between
        for sample in (True, False):
            both(n, 5, sample)
            both(n, 5, sample)
        both(1 + n % 3, 6, True)
    assert made() == 3
    for pos in range(64, 128):   # one, then two tiles of keys: one more kind at most
        both(2, pos, True)
    assert made() <= 4


def test_held_results_stay_as_they_were():
    """Results are handed out in buffers that later calls use again: not while a caller still holds an array, a view or a tensor of them."""
    from ssd_b200 import hybrid_bench as hb
    from ssd_b200.hybrid import HybridRunner, random_hybrid_weights
    spec = hb.kokatar_spec(dict(hb.SIZES["s"], layers=1, vocab=512))
    r = HybridRunner(spec, random_hybrid_weights(spec, torch.bfloat16, "cuda:0", seed=2), max_tokens=64, max_seqs=9, block_size=64, num_blocks=9, n_slots=9, max_model_len=64)
    assert all(buf.size == 9 * 512 for buf in r._pinned)   # a row per sequence
    call = lambda k: r.forward([([k + i], 0, i, [i], [0]) for i in range(9)])[0]
    held, copies = [], []
    for k, keep in enumerate((lambda a: a, lambda a: a[3:5], lambda a: torch.from_numpy(a), lambda a: a.T, lambda a: memoryview(a), lambda a: a.reshape(-1)[::2])):
        got = keep(call(20 * k))
        held.append(got)
        copies.append(np.asarray(got).copy())
    for k in range(4):
        call(300 + k)
    for a, b in zip(held, copies):
        assert np.array_equal(np.asarray(a), b)
    pinned = [buf.ctypes.data for buf in r._pinned]
    del held, got, a
    assert call(1).ctypes.data in pinned   # and they come back once nobody holds them
