"""Logits of several places of a portion, computed together, against the same places one at a time (the one-row kernel, f32)."""
import numpy as np
import pytest

import virolorn_util as vu

pytestmark = pytest.mark.gpu

_cfg = vu.config([vu.lightning()], width=192, vocab=301)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("count", [2, 7, 8, 9, 16, 17, 32, 33, 65])
def test_places_together_and_one_by_one(dev, dtype, count):
    n = 70
    w, t = vu.weights(_cfg), vu.tokens(_cfg, n, 3)
    places = np.sort(np.random.default_rng(count).permutation(n)[:count]).tolist()
    m = vu.build(dev, _cfg, w, n, dtype=dtype)
    one = []
    for p in places:
        one.append(m.extend(t, [p])[0])
        m.release(0)
    got = m.extend(t, places)
    # f32 sums of 192 products in another order: 192 * 2^-24 of the row at most, less than an eighth of it in practice (1.4e-6; with
    # two of the three bf16 terms of the rows the products would be off by 3.1e-6)
    assert vu.row_errors(got, np.stack(one)).max() < 192 * 2.0 ** -24 / 8
    assert np.array_equal(m.read_logits(_cfg["vocab"]).ravel(), got[-1])
    m.destroy()


@pytest.mark.parametrize("max_seq,max_rows,own", [(600, 0, 0), (35, 0, 1), (600, 5, 1)])
def test_memory_of_the_places(dev, max_seq, max_rows, own):
    """The logits of several places go where the portion's activations were; only blocks of few rows have a buffer for them."""
    places, made = [0, 3, 4, 5, 17, 20, 21, 33, 34], []
    for width in (63, 64):  # (no such logits where the width is no multiple of 64)
        cfg = vu.config([vu.lightning(mlp={"kind": "dense", "ff": 24})], width=width, vocab=4000)
        w, t = vu.weights(cfg), vu.tokens(cfg, 35, 3)
        before = dev.pool_stats()
        m = vu.build(dev, cfg, w, max_seq, max_rows=max_rows)
        held = dev.pool_stats()
        made.append(held["allocations"] + held["reuses"] - before["allocations"] - before["reuses"])
        one = []
        for p in places:
            one.append(m.extend(t, [p])[0])
            m.release(0)
        got = m.extend(t, places)
        assert dev.pool_stats()["bytes_in_use"] == held["bytes_in_use"]
        assert vu.row_errors(got, np.stack(one)).max() < 64 * 2.0 ** -24 / 4
        m.destroy()
    assert made[1] == made[0] + own


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_what_follows_does_not_depend_on_wanted_places(dev, dtype):
    """Portions and steps behind one whose places were wanted: bit for bit those behind one that wanted none (odd inner sizes: rows
    with padding)."""
    cfg = vu.config([vu.delta(heads=3, kv_heads=3, dim=20, vdim=13, ranks=(6, 11), mlp={"kind": "dense", "ff": 27}), vu.lightning(heads=3, dim=21, vdim=13),
                     vu.latent(heads=3, dim=13, rot_dim=10, vdim=9, kv_rank=37, q_rank=29, mlp={"kind": "dense", "ff": 45})], width=64, vocab=301)
    w, t = vu.weights(cfg), vu.tokens(cfg, 140, 3)
    m = vu.build(dev, cfg, w, 140, dtype=dtype)
    seen = []
    for want in ((), range(0, 60, 3)):
        m.release(0)
        m.extend(t[:60], want)
        out = [m.extend(t[60:130], [69])]
        for x in t[130:]:
            m.decode([x], 1)
            out.append(m.read_logits(cfg["vocab"]))
        seen.append(np.concatenate([np.ravel(x) for x in out]))
    assert np.isfinite(seen[0]).all() and np.array_equal(*seen)
    m.destroy()
