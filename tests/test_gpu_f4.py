"""The tcgen05 wave counter (csrc/count_f4.cu) at the edges of its tiles: row groups of 16 and
256, column tiles of 128, narrow tiles of one, two and four chunks per stage, word slices of one
block, and full accumulators.  Supports are whole numbers: every comparison is exact."""
import numpy as np
import pytest

import tensorfim_b200 as tf

pytestmark = pytest.mark.gpu


def _bits(rows, n_bits, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    x = rng.integers(0, 2 ** 32, size=(rows, (n_bits + 31) // 32), dtype=np.uint64).astype(np.uint32)
    if n_bits % 32:
        x[:, -1] &= np.uint32((1 << (n_bits % 32)) - 1)
    return x


@pytest.mark.parametrize("b,d,n_bits", [(1, 1, 1), (3, 7, 2048), (16, 72, 2049), (17, 8, 40_000), (96, 129, 70_001),
                                        (97, 128, 4096), (255, 40, 10_007), (256, 127, 6_000), (257, 257, 9_999),
                                        (640, 3, 33_333)])
def test_tile_edges(oracle_mod, b, d, n_bits):
    rows = _bits(d, n_bits, seed=b + d)
    rng = np.random.Generator(np.random.PCG64(b * 1000 + d))
    lists = [[int(v) for v in rng.integers(0, d, size=int(rng.integers(0, 4)))] for _ in range(b)]
    ref_c, ref_n = oracle_mod.count_wave(rows, lists, d, n_bits // 4)
    with tf.Database.from_bitmap(rows, n_bits, d) as db:
        for counter in ("i8", "auto"):
            got_c, got_n = db.count_wave(lists, n_bits // 4, counter=counter)
            assert (got_c == ref_c).all(), np.argwhere(got_c != ref_c)[:5]
            assert (got_n == ref_n).all()


@pytest.mark.parametrize("n_bits", [(1 << 23) - 1, 1 << 23, (1 << 24) + 65])
def test_full_accumulators(n_bits):
    """Every transaction holds every item: each count is the number of transactions, which a
    tile's FP32 sum reaches one by one up to its 2^23 transactions."""
    d, b = 130, 17
    rows = np.full((d, (n_bits + 31) // 32), 0xFFFFFFFF, np.uint32)
    if n_bits % 32:
        rows[:, -1] = (1 << (n_bits % 32)) - 1
    with tf.Database.from_bitmap(rows, n_bits, d) as db:
        counts, nfreq = db.count_wave([[i, 2 * i] for i in range(b)], n_bits, counter="i8")
    assert (counts == n_bits).all() and (nfreq == d).all()
