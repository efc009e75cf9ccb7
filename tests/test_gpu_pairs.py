"""Products in tiles that two SMs share (gemm_bf16.cu), every width that is picked (128 only where K is long, which latents and decays do not
have) and every kind of result, through one layer against the plain oracle."""
import numpy as np
import pytest

import fenorax_util as fu
import hybrid_oracle as ho
import virolorn_oracle as vo
import virolorn_util as vu
from tiles_rule import pick

pytestmark = pytest.mark.gpu
TOL, RMS = 8e-2, 3.5e-2  # row errors of bf16 activations, as in test_gpu_fenorax.py


def through(dev, util, oracle, cfg, rows, product, bn):
    assert pick(rows, *product) == (bn, True)
    w, t = util.weights(cfg), util.tokens(cfg, rows)
    want = oracle.forward(cfg, util.values(w), t)[0]
    m = util.build(dev, cfg, w, rows, dtype="bfloat16")
    err = util.row_errors(m.extend(t, range(rows)), want)
    m.destroy()
    assert err.max() < TOL and np.sqrt((err ** 2).mean()) < RMS, (err.max(), int(err.argmax()))


# (the last two: several tiles of rows, the last of them ends in the first SM's half)
@pytest.mark.parametrize("rows,ff,width,bn", [(120, 4904, 4096, 128), (148, 4904, 1536, 160), (187, 4904, 1024, 192), (220, 4904, 768, 224), (247, 4904, 768, 256), (868, 2704, 1024, 160), (1130, 1560, 1024, 256)])
def test_gated_results(dev, rows, ff, width, bn):
    cfg = fu.config([fu.attention(heads=2, kv_heads=1, dim=32, vdim=32, chunk=50, mlp={"kind": "dense", "ff": ff, "limit": 1.0})], width=width)
    through(dev, fu, ho, cfg, rows, (2 * ff, width), bn)


@pytest.mark.parametrize("rows,heads,width,bn", [(117, 150, 4096, 128), (148, 150, 1536, 160), (187, 151, 1024, 192), (220, 150, 768, 224), (247, 151, 768, 256), (1018, 35, 1536, 160), (776, 56, 1536, 224)])
def test_32_bit_results(dev, rows, heads, width, bn):
    cfg = fu.config([fu.attention(heads=heads, kv_heads=1, dim=64, vdim=64, scale=0.3, chunk=50, mlp=None)], width=width)
    through(dev, fu, ho, cfg, rows, (heads * 64 + 128 + heads, width), bn)


@pytest.mark.parametrize("rows,kv_rank,heads,bn", [(777, 768, 56, 160), (187, 768, 76, 192), (211, 512, 76, 224), (246, 448, 76, 256)])
def test_16_bit_results(dev, rows, kv_rank, heads, bn):
    """Keys and values of all heads formed from the latents."""
    cfg = vu.config([vu.latent(heads=heads, dim=128, rot_dim=64, vdim=128, kv_rank=kv_rank, q_rank=32, scale=0.07)], width=128)
    through(dev, vu, vo, cfg, rows, (heads * 256, kv_rank), bn)


@pytest.mark.parametrize("rows,rank,bn", [(150, 1024, 160), (187, 768, 192), (211, 512, 224), (246, 448, 256)])
def test_decays(dev, rows, rank, bn):
    cfg = vu.config([vu.delta(heads=152, kv_heads=8, dim=128, vdim=8, ranks=(rank, 10))], width=128)
    through(dev, vu, vo, cfg, rows, (152 * 128, rank), bn)
