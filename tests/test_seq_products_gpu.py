"""Matrix products of the layer-list library at the edges of their kernels' ranges, against float64 products of the same operands."""
import numpy as np
import pytest

import gtb  # noqa: F401
from tinyllama_cpp_b200 import safetensors_io as st
from tinyllama_cpp_b200 import seq

pytestmark = pytest.mark.gpu


def operands(M, N, K, seed):
    rng = np.random.default_rng(seed)
    bits = [st.f32_to_bf16_bits(rng.standard_normal(s, np.float32)) for s in ((M, K), (N, K))]
    f = [(b.astype(np.uint32) << 16).view(np.float32) for b in bits]
    return bits, f, rng.standard_normal((M, N), np.float32)


# row counts around the tile sizes of the split-K kernel (16, 32, 64) and the switch to the persistent one; columns around its 128-wide
# tiles, unaligned rows of C among them; K of one block, of fewer blocks than CTAs in a cluster, and of uneven shares
@pytest.mark.parametrize("M,N,K", [
    (1, 16, 64), (9, 1, 64), (16, 128, 192), (17, 129, 448), (31, 100, 2048), (32, 2048, 64), (33, 6400, 128), (48, 127, 1024), (63, 257, 704),
    (64, 64, 4096), (65, 384, 320), (100, 2047, 2048), (128, 5003, 64), (129, 96, 1088), (256, 640, 512), (400, 1000, 192), (513, 4100, 128), (700, 130, 64), (2048, 19, 128),
])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_product(M, N, K, accumulate):
    seq.init(0)
    (ab, wb), (a, w), c0 = operands(M, N, K, M * 7 + N)
    got, _ = seq.selftest_gemm(ab, wb, c0 if accumulate else None, ld_extra=8)
    want = a.astype(np.float64) @ w.astype(np.float64).T + (c0 if accumulate else 0.0)
    # products of bf16 values are exact in fp32; every addition rounds (or cuts off) at most one unit of the running sum's last place,
    # and no running sum is larger than the sum of the magnitudes
    bound = (K + 8) * 2.0 ** -23 * (np.abs(a).astype(np.float64) @ np.abs(w).astype(np.float64).T + np.abs(c0))
    assert got.shape == want.shape
    assert np.all(np.abs(got - want) <= bound)


def test_float32_products_on_bf16_pieces():
    """float32 mode: products of nine rows and more run on three exact bf16 pieces per value; no further from float64 than the FFMA kernels."""
    from oracle import seq_ref as R
    from tinyllama_cpp_b200 import reninex
    seq.init(0)
    cfg = reninex.make_config(vocab=96, width=160, n_layers=2, ff=416, taps=3, l_heads=4, l_kv=2, l_dim=24, l_vdim=40, r_heads=2, r_dim=32, r_vdim=40, rot_dims=16, loop=(0, 1, 2))
    desc = reninex.describe(cfg)
    t = reninex.synth_tensors(desc, 11, gain=1.5)
    W = {k: R.bf16_to_float(v) for k, v in t.items()}
    toks = np.random.default_rng(3).integers(0, 96, 300).astype(np.int32)
    want = R.forward(cfg, W, toks)[0]
    err = {}
    for tensor in (1, 0):
        m = seq.SeqModel(desc, seq.F32, 1, 320, max_rows=128).load(t)           # 300 rows in passes of 128
        m.set_option("tensor", tensor)
        got = np.concatenate([m.step([(0, toks[:9])], range(9)), m.step([(0, toks[9:40])], range(31)), m.step([(0, toks[40:])], range(260))])
        err[tensor] = np.linalg.norm(got - want) / np.linalg.norm(want)
        m.close()
    assert err[1] < 1.2 * err[0] + 1e-7, err
