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


@pytest.mark.parametrize("max_rows,vocab", [(0, 4000), (0, 20000), (5, 20000)])
def test_no_memory_of_their_own(dev, max_rows, vocab):
    """The logits of several places go where the portion's activations were: as many at a time as fit there (all, 4, none)."""
    cfg = vu.config([vu.lightning(mlp={"kind": "dense", "ff": 2400})], width=64, vocab=vocab)
    w, t = vu.weights(cfg), vu.tokens(cfg, 35, 3)
    places = [0, 3, 4, 5, 17, 20, 21, 33, 34]
    m = vu.build(dev, cfg, w, 35, max_rows=max_rows)
    one = []
    for p in places:
        one.append(m.extend(t, [p])[0])
        m.release(0)
    held = dev.pool_stats()["bytes_in_use"]
    got = m.extend(t, places)
    assert dev.pool_stats()["bytes_in_use"] == held
    assert vu.row_errors(got, np.stack(one)).max() < 64 * 2.0 ** -24 / 4
    hidden = m.read_hidden(min(max_rows or 35, 35))
    m.release(0)
    m.extend(t)  # the same hidden rows as without wanted places
    assert np.array_equal(m.read_hidden(hidden.shape[0]), hidden)
    m.destroy()
