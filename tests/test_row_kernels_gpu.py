"""Row kernels of the recurrent mixers that take four channels (and several rows) per thread, against the float64 oracle in 32 bits: prompts long enough for
them whose rows belong to several sequences, portions shorter than the convolution behind earlier ones, channels around a block of threads."""
import numpy as np
import pytest
import torch

from tests import kefurax_util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layer,width", [
    (U.mamba1(inner=520, state=8, dt_rank=8, conv=4), 64),
    (U.rglru(width=528, blocks=4, conv=4), 64),
    (U.parallel(left=U.attention(heads=4, kv_heads=2, dim=64, vdim=24, dims=32), right=U.delta(heads=2, kv_heads=1, dim=16, vdim=128, conv=4)), 64),
    (U.parallel(left=U.attention(heads=3, kv_heads=1, dim=128, vdim=132, dims=4), right=U.delta(heads=1, kv_heads=1, dim=8, vdim=128, conv=2)), 48)])
def test_against_the_oracle(tmp_path, layer, width):
    from ssd_b200.hybrid import HybridRunner, HybridSpec, load_hybrid_weights
    cfg = U.config([layer], width=width)
    tensors = U.random_tensors(cfg, 2)
    path = U.write_checkpoint(str(tmp_path / "c"), cfg, tensors)
    spec = HybridSpec.from_dir(path)
    r = HybridRunner(spec, load_hybrid_weights(path, spec, torch.float32, "cuda:0"), dtype="float32", max_tokens=1024, max_seqs=3, block_size=16, num_blocks=96, n_slots=3,
                     max_model_len=512)
    toks = [torch.randint(0, cfg["vocab"], (n,), generator=torch.Generator().manual_seed(n)).tolist() for n in (260, 190, 150)]
    want = [U.PlainModel(cfg, tensors).run(t).numpy() for t in toks]
    pages = [list(range(i * 32, (i + 1) * 32)) for i in range(3)]
    at = [0, 0, 0]
    for part in ((129, 1, 2), (2, 127, 1), (1, 2, 146), (128, 60, 1)):
        entries = [(toks[i][at[i]:at[i] + n], at[i], i, pages[i], list(range(n))) for i, n in enumerate(part)]
        got, row = r.forward(entries)[0], 0
        for i, n in enumerate(part):
            # (fp32 sums of a few hundred terms in a handful of products: 1e-6 .. 1e-5; a row or a tap out of place shows as 1e-2 and more)
            assert U.rel_err(got[row:row + n], want[i][at[i]:at[i] + n]) < 3e-5, (part, i)
            row += n
        at = [x + n for x, n in zip(at, part)]
