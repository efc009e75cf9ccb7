"""Sizes that the tensor-core kernels ask of an MMA, over the ranges their callers have."""
import random

from tiles_rule import columns, pick


def test_16_bit_products_ask_for_widths_that_exist():
    """One CTA (128 features): 16 to 256 columns in steps of 16; two (256 features): 32 to 256 in steps of 32."""
    rng, widths = random.Random(1), {True: set(), False: set()}
    for _ in range(20000):
        m, n, k = rng.randint(2, 4096), rng.randint(16, 32768), rng.choice([24, 64, 256, 768, 1024, 4096, 12288])
        bn, pair = pick(m, n, k, sms=rng.choice([148, 132, 2]))
        widths[pair].add(bn)
        assert bn % (32 if pair else 16) == 0 and 16 <= bn <= 256, (m, n, k, bn, pair)
        assert not pick(m, n, k, may_pair=False)[1]
    assert widths[True] == {128, 160, 192, 224, 256}  # (the widths that tests of pairs have to reach)


def test_q4k_pairs_ask_for_widths_that_exist():
    taken = set()
    for n in range(128, 65537, 128):
        for m in (257, 512, 700, 1024, 1500, 2048, 4096):
            cols, wide_tiles, wide, narrow = columns(m, n)
            if not cols:
                continue
            taken |= {narrow, wide} if wide_tiles else {narrow}
            assert narrow % 32 == 0 and wide == narrow + 32 and 128 <= narrow and 0 <= wide_tiles < cols
            assert (cols - wide_tiles) * narrow + wide_tiles * wide == n
    assert {128, 160, 192, 224, 256} <= taken
