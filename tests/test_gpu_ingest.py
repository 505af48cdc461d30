"""The bitmap built from the transaction list (csrc/ingest.cu) at the edges of its blocks: 256 and
512 rows, and tables of up to 700 items (64-byte pieces), up to 6,400 (32-byte pieces) and
beyond (global atomics).  Supports of single items and pairs are exact."""
import numpy as np
import pytest

import tensorfim_b200 as tf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,items", [(1, 1), (255, 40), (256, 700), (257, 701), (511, 9), (512, 700), (513, 1500),
                                        (5000, 64), (700, 6400), (700, 6401), (2049, 300)])
def test_bitmap_edges(rows, items):
    rng = np.random.Generator(np.random.PCG64(rows * 10_007 + items))
    lens = rng.integers(0, 24, size=rows)
    lens[rng.integers(0, rows)] = 30
    held = [np.sort(rng.choice(items, size=min(int(m), items), replace=False)) + 1 for m in lens]
    held[0] = np.arange(1, items + 1)   # every item occurs
    off = np.concatenate([[0], np.cumsum([len(h) for h in held])]).astype(np.int64)
    flat = np.concatenate(held).astype(np.int32)
    on = np.zeros((items + 1, rows), dtype=bool)
    on[flat, np.repeat(np.arange(rows), np.diff(off))] = True
    some = rng.integers(0, items, size=min(items, 40))
    with tf.Database.from_csr(off, flat, 0.5 / rows) as db:
        assert db.info["n_dense"] == items and db.info["trans_num_reduced"] == int(on.any(0).sum())
        counts, _ = db.count_wave([[]] + [[int(i)] for i in some], 1, counter="lop3")
    assert (counts[0] == on[1:].sum(1)).all()
    for i, row in zip(some, counts[1:]):
        assert (row == (on[1:] & on[i + 1]).sum(1)).all()
