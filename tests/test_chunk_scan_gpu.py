"""Portions of many rows through the recurrences walked in pieces (rglru_chunk_scan_kernel, selective_chunk_scan_kernel) against the float64
oracle: row counts around the switch and the pieces' edges, carried states, states that fill a lane's registers or not."""
import numpy as np
import pytest
import torch

from tests import kefurax_util as U

pytestmark = pytest.mark.gpu

TOL = 1e-4   # fp32 through two projections and a recurrence of some hundred steps (rounding 1e-6); a lost piece or state is 1e-2 and more


@pytest.mark.parametrize("layer", [U.rglru(width=34, blocks=2), U.mamba1(inner=33, state=6, dt_rank=3), U.mamba1(inner=40, state=8, dt_rank=4),
                                   U.mamba1(inner=31, state=16, dt_rank=4), U.mamba1(inner=64, state=13, dt_rank=5)],
                         ids=["rglru", "state-6", "state-8", "state-16", "state-13"])
def test_pieces_match_the_oracle(tmp_path, layer):
    from ssd_b200.hybrid import HybridRunner, HybridSpec, load_hybrid_weights
    cfg = U.config([layer])
    tensors = U.random_tensors(cfg, 4)
    path = U.write_checkpoint(str(tmp_path / "ckpt"), cfg, tensors)
    spec = HybridSpec.from_dir(path)
    r = HybridRunner(spec, load_hybrid_weights(path, spec, torch.float32, "cuda:0"), dtype="float32", max_tokens=600, max_seqs=2, block_size=16, num_blocks=40, n_slots=2, max_model_len=640)
    plain = U.PlainModel(cfg, tensors)
    toks = torch.randint(0, cfg["vocab"], (290,), generator=torch.Generator().manual_seed(1)).tolist()
    want = plain.run(toks).numpy()
    for cuts in ([290], [63, 64, 65, 98], [1, 127, 2, 97, 63], [200, 90]):
        got, at = [], 0
        for n in cuts:   # the other slot's sequence runs a prompt of its own beside it
            other = (toks[:max(1, n // 3)], 0, 0, [], [])
            got.append(r.forward([(toks[at:at + n], at, 1, [], list(range(n))), other])[0])
            at += n
        assert U.rel_err(np.concatenate(got), want) < TOL, cuts
