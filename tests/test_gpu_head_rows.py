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
    # f32 sums of 192 products in another order: 192 * 2^-24 of the row at most, an eighth of it in practice
    assert vu.row_errors(got, np.stack(one)).max() < 192 * 2.0 ** -24
    assert np.array_equal(m.read_logits(_cfg["vocab"]).ravel(), got[-1])
    m.destroy()
