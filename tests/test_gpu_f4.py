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


def _slice_words(nodes, items, words, sms=148):
    """The words of a tile of the wave counter (tiles_f4), restated."""
    groups = -(-nodes // 256)
    step = (-(-nodes // groups) + 15) & ~15
    base = -(-nodes // step) * -(-items // 128)
    blocks = words // 64
    best = None
    for ks in range(1, min(blocks, max(1, 4 * sms // base) + (words >> 18) + 1) + 1):
        per = -(-blocks // ks)
        if per * 64 <= 1 << 18:
            cost = -(-base * -(-blocks // per) // sms) * (per * 4 + 16)
            if best is None or cost < best[0]:
                best = cost, per
    return best[1] * 64


def test_longest_slice():
    """37 row groups x 4 column tiles fill the 148 SMs once, so a tile takes all of 2^23 transactions:
    its FP32 sums reach 2^23.  Items hold every transaction but some of the first 4,096."""
    n, d, b = 1 << 23, 512, 37 * 256
    assert _slice_words(b, d, n // 32) == n // 32
    rng = np.random.Generator(np.random.PCG64(3))
    head = rng.random((d, 4096)) < rng.random((d, 1))
    head[:3] = True
    rows = np.full((d, n // 32), 0xFFFFFFFF, np.uint32)
    rows[:, :128] = np.packbits(head, axis=1, bitorder="little").view(np.uint32)
    lists = [[k % d, (k * 7 + k // d) % d] for k in range(b)]
    both = np.array([head[i] & head[j] for i, j in lists], np.float32)
    expected = (both @ head.T.astype(np.float32)).astype(np.int64) + n - 4096
    with tf.Database.from_bitmap(rows, n, d) as db:
        counts, nfreq = db.count_wave(lists, n, counter="i8")
    assert (counts == expected).all() and (nfreq == (expected >= n).sum(1)).all()
    assert counts.max() == n
