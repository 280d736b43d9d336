"""Chunked retention with value heads wider than 64 channels against the row-by-row walk and the float64 restatement: chunks that end early, value
slices that are not full, head sizes below and at the tiles' width."""
import numpy as np
import pytest

import gtb  # noqa: F401
from oracle import seq_ref as R
from tinyllama_cpp_b200 import reninex, seq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r_dim,r_vdim,rot", [(128, 128, 64), (64, 128, 0), (4, 68, 4), (100, 132, 36), (128, 260, 128), (32, 72, 0)])
@pytest.mark.parametrize("mode,tol", [("float32", 1e-5), ("bfloat16", 3e-2)])
def test_wide_value_heads(r_dim, r_vdim, rot, mode, tol):
    seq.init(0)
    cfg = reninex.make_config(vocab=48, width=64, n_layers=1, ff=64, taps=2, l_heads=2, l_kv=1, l_dim=16, l_vdim=16, r_heads=3, r_dim=r_dim, r_vdim=r_vdim, rot_dims=rot)
    desc = reninex.describe(cfg)
    t = reninex.synth_tensors(desc, 5)
    W = {k: R.bf16_to_float(v) for k, v in t.items()}
    rng = np.random.default_rng(1)
    a, b = rng.integers(0, 48, 215).astype(np.int32), rng.integers(0, 48, 64).astype(np.int32)
    m = seq.SeqModel(desc, seq.MODE_BY_NAME[mode], 2, 300).load(t)
    g1 = m.step([(0, a[:65])], range(65))                              # a chunk and one row
    g2 = m.step([(1, b), (0, a[65:150])], range(64 + 85))              # exactly one chunk beside one that ends early
    g3 = m.step([(0, a[150:])], range(65))
    got = [np.concatenate([g1, g2[64:], g3]), g2[:64]]
    for g, toks in zip(got, (a, b)):
        want = R.forward(cfg, W, toks)[0]
        assert np.linalg.norm(g - want) < tol * np.linalg.norm(want)
    m.close()
