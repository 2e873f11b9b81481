"""Host side of sampled prompts: whatever a pass carries, a prompt's first token is drawn with the numbers that calls of 256 tokens give it,
the calls that follow keep theirs, and a chunk that a caller asks for bounds every pass."""
import random

from ssd_b200.runner import PairRunner


class Rec:
    """The planners on a recorder of calls: (call number, row) of every prompt's sampling call, and the widest call."""
    plan_prefill_call = staticmethod(PairRunner.plan_prefill_call)
    draw_numbers = staticmethod(PairRunner.draw_numbers)
    prefill_many = PairRunner.prefill_many
    prefill = PairRunner.prefill

    def __init__(self, most, max_batch=8):
        self.most, self.max_batch, self.step_id, self.drawn, self.widest, self.calls = most, max_batch, 100, {}, 0, 0

    def pass_tokens(self, which):
        return self.most

    def forward_tokens(self, which, ids, ctx_len, block_tables, temps=None, want_sample=True, seed=0, *, rows=256, draws=None):
        B, Q = len(ids), len(ids[0])
        assert B * Q <= max(rows, 256)
        self.widest, self.calls = max(self.widest, B * Q), self.calls + 1
        if draws is None:
            if rows > 256:
                self.step_id += max(0, -(-B * Q // 256) - 1)
            draws = [(self.step_id, b) for b in range(B)]
            self.step_id += 1
        for b, (table, x) in enumerate(zip(block_tables, ids)):
            self.drawn[table[0]] = draws[b]   # (the last call of a prompt stays)
        return [x[-1] for x in ids] if want_sample else None


def test_draws_are_those_of_short_calls():
    rng = random.Random(7)
    for trial in range(60):
        n, batch = rng.randint(1, 9), rng.randint(1, 8)
        lens = [rng.choice([1, 7, 100, 128, 255, 256, 257, 300, 517, 2000, 2049]) for _ in range(n)]
        starts = [rng.choice([0, 0, 0, min(256, l - 1)]) for l in lens]
        toks, tables = [[0] * l for l in lens], [[i] for i in range(n)]
        short, long = Rec(256, batch), Rec(2048, batch)
        for r in (short, long):
            r.prefill_many(0, toks, tables, starts, temps=[0.7] * n)
        assert long.drawn == short.drawn and long.step_id == short.step_id, (lens, starts, batch)
        assert long.calls <= short.calls


def test_a_chunk_bounds_every_pass():
    for chunk in (1, 64, 255, 256):
        r = Rec(2048)
        r.prefill(0, [0] * 1000, [0], chunk=chunk)
        assert r.widest == chunk
        r = Rec(2048)
        r.prefill_many(0, [[0] * 1000, [0] * 999], [[0], [1]], [0, 0], chunk=chunk)
        assert r.widest <= chunk
    r = Rec(2048)
    r.prefill(0, [0] * 1000, [0])
    assert r.widest == 1000
