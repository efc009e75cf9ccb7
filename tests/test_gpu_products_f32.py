"""32-bit mode: products of several rows on the tensor cores as three bf16 terms (csrc/gemm_bf16w_f32.cu), through one-layer
decoders sized so that every tile width, several tiles per CTA, long and short K and remainders in M, N and K occur.  The
tolerance tells f32 from two terms: with the third one lost, the rows are off by 1.2e-5."""
import numpy as np
import pytest

import virolorn_oracle as vo
from virolorn_util import build, config, delta, latent, lightning, row_errors, tokens, values, weights

pytestmark = pytest.mark.gpu


def ff(n):
    return {"kind": "dense", "ff": n}


# 333 rows (11, 6, 4, 3 tiles of 32, 64, 96, 128); features of the widest product -> width of its tiles on 148 SMs
CASES = {
    "32 wide": config([lightning(heads=3, dim=40, vdim=52, mlp=ff(136))], width=200),                       # 572 -> 32
    "64 wide, odd width": config([lightning(heads=4, dim=33, vdim=70, mlp=ff(1100))], width=203),            # 2200 -> 64
    "96 wide": config([lightning(heads=2, dim=64, vdim=64, mlp=ff(2005))], width=264),                       # 4010 -> 96
    "128 wide, three stages": config([lightning(heads=2, dim=64, vdim=64, mlp=ff(2796))], width=320),        # 5592 -> 128
    "several tiles per CTA": config([lightning(heads=2, dim=64, vdim=64, mlp=ff(6003))], width=513),         # 12006, K 513 and 6003
    "decay": config([delta(heads=17, kv_heads=17, dim=120, vdim=20, ranks=(70, 3))], width=129),             # 2040 decays, K 70
    "decay of few rows": config([delta(heads=6, kv_heads=3, dim=36, vdim=40, ranks=(129, 65), mlp=ff(24))], width=72),
    "latent": config([latent(heads=9, dim=40, rot_dim=16, vdim=36, kv_rank=72, q_rank=130, mlp=ff(96))], width=136),
}


@pytest.mark.parametrize("rows", [2, 33, 333])
@pytest.mark.parametrize("name", CASES)
def test_rows_against_64_bits(dev, name, rows):
    cfg = CASES[name]
    w = weights(cfg)
    t = tokens(cfg, rows, 5)
    logits, res = vo.forward(cfg, values(w), t)
    m = build(dev, cfg, w, rows)
    got = m.extend(t, range(rows))
    err = np.concatenate([row_errors(got, logits), row_errors(m.read_hidden(rows), res[-1])])
    assert np.sqrt((err ** 2).mean()) < 1e-6 and err.max() < 4e-6, (err.max(), np.sqrt((err ** 2).mean()))
    m.destroy()
