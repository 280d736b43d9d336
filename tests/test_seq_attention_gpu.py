"""Tensor-core attention of prompt portions (head sizes 64 and 128) against the row-at-a-time kernels (fp32 weights) on the same bf16 operands:
every mask and option the tiled kernel takes, portions that end at, before and behind the borders of its 128-row and 64- / 128-key tiles."""
import numpy as np
import pytest

import gtb  # noqa: F401
from tinyllama_cpp_b200 import bisodra, nanotar, reninex, robopel, seq, vulosun

pytestmark = pytest.mark.gpu


def vul(dim, vdim, **kw):
    return vulosun, vulosun.make_config(vocab=64, width=64, layers=[vulosun.gated_attention_layer(heads=4, kv_heads=2, dim=dim, vdim=vdim, rot_dims=16, **kw)])


CASES = {
    "causal_64_64": lambda: vul(64, 64),
    "causal_64_128": lambda: vul(64, 128),
    "causal_128_64": lambda: vul(128, 64),
    "causal_128_128": lambda: vul(128, 128),
    "negative_scale": lambda: vul(64, 64, scale=-0.3),
    "sharp_scores": lambda: vul(64, 64, scale=6.0),                    # the reference maximum moves again and again
    "two_maps_in_chunks": lambda: (vulosun, vulosun.make_config(vocab=64, width=64, layers=[vulosun.differential_layer(heads=2, kv_heads=1, dim=64, vdim=128, chunk=150, rot_dims=16)])),
    "sink_beside_recurrence": lambda: (vulosun, vulosun.make_config(vocab=64, width=64, layers=[vulosun.parallel_layer(heads=4, kv_heads=2, dim=128, vdim=128)])),
    "window_with_sink": lambda: (nanotar, nanotar.make_config(vocab=64, width=64, layers=[nanotar.latent_layer(heads=2, dim=48, rot_dim=16, vdim=64, kv_rank=64, q_rank=32, window=100, mlp=None)])),
    "latent_128": lambda: (nanotar, nanotar.make_config(vocab=64, width=64, layers=[nanotar.latent_layer(heads=2, dim=96, rot_dim=32, vdim=128, kv_rank=64, mlp=None)])),
    "sigmoid_64": lambda: (reninex, reninex.make_config(vocab=64, width=64, n_layers=1, l_heads=4, l_kv=1, l_dim=64, l_vdim=64)),
    "sigmoid_128_64": lambda: (reninex, reninex.make_config(vocab=64, width=64, n_layers=1, l_heads=2, l_kv=2, l_dim=128, l_vdim=64)),
    "soft_capped_window": lambda: (robopel, robopel.make_config(vocab=64, width=64, layers=[robopel.attention_layer(heads=4, kv_heads=2, dim=64, vdim=64, window=140, pool=0, softcap=5.0)])),
    "slopes_keys_as_values": lambda: (bisodra, bisodra.make_config(vocab=64, width=64, layers=[bisodra.windowed_layer(heads=2, kv_heads=1, dim=64, window=90, keep_first=0)])),
}


@pytest.mark.parametrize("name", list(CASES))
def test_tiles_match_row_kernels(name):
    seq.init(0)
    fam, cfg = CASES[name]()
    desc = fam.describe(cfg)
    m = seq.SeqModel(desc, seq.BF16, 4, 700).load(fam.synth_tensors(desc, 3, gain=2.0))
    rng = np.random.default_rng(5)
    a, b, c = (rng.integers(0, 64, n).astype(np.int32) for n in (600, 257, 128))

    def passes():
        for s in range(3):
            m.reset(s)
        out = [m.step([(0, a[:127]), (2, c)], range(127 + 128))]                   # one row short of a tile beside a whole one
        out.append(m.step([(0, a[127:256]), (1, b)], range(129 + 257)))            # starts at 127: tiles of a later portion do not start on tile borders
        out.append(m.step([(0, a[256:600])], range(344)))
        return np.concatenate(out)
    got = passes()
    m.set_option("fused_attn", 0)
    want = passes()
    # bf16 weights (2^-9 each, averaged over the keys) and bf16 rounding of differing fp32 results in what follows the layer
    assert np.linalg.norm(got - want) < 1e-2 * np.linalg.norm(want)
    assert np.abs(got - want).max() < 0.1 * np.abs(want).max()
    m.close()


def test_rows_behind_a_sequence_do_not_leak():
    """A slot that held infinities and is used again: its stale cache rows lie inside the new sequence's last key tile."""
    seq.init(0)
    fam, cfg = vul(64, 64)
    desc = fam.describe(cfg)
    t = fam.synth_tensors(desc, 3, gain=2.0)
    m = seq.SeqModel(desc, seq.BF16, 2, 400).load(t)
    rng = np.random.default_rng(7)
    a = rng.integers(1, 64, 200).astype(np.int32)
    want = m.step([(1, a[:150])], range(150))
    bad = t["embed"].copy().reshape(64, 64)
    bad[0] = 0x7F80                                                                # token 0: infinities
    m.set_tensor("embed", bad)
    m.step([(0, np.concatenate([a[:150], np.zeros(50, np.int32)]))], [199])
    m.reset(0)
    assert np.array_equal(m.step([(0, a[:150])], range(150)), want)
    m.close()
