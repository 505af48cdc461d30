"""Kernels at the edges of their tiles and tables: the packed tensor-core counter's column classes
(csrc/count_pk.cu), the result sort of a mine on the device (csrc/resident.cu, up to 4,096 sets), and the
dense-id tables (csrc/ingest.cu, up to 32,768 items).  Every value is an exact integer."""
import numpy as np
import pytest

import tensorfim_b200 as tf

pytestmark = pytest.mark.gpu


def _csr(hit):
    row, item = np.nonzero(hit)
    return np.concatenate([[0], np.cumsum(hit.sum(1))]).astype(np.int64), (item + 1).astype(np.int32)


# Clusters of items, each in half of the transactions and its items in half of those, and a threshold
# between the supports of pairs (1/8) and of triples and pairs across clusters (1/16): the families
# have as many columns as their cluster has other items.  Widths 9, 17, 25, 33, 41 and 65 open a new
# class of tiles, 129 is too wide for one.
@pytest.mark.parametrize("rows,opts", [(20_011, dict(counter="i8")), (33_000, dict(counter="i8", small_pools=True)),
                                       (20_011, dict(counter="i8", wave_cap=70)), (140_003, dict())])
def test_packed_tiles_of_every_width(rows, opts):
    sizes = [2, 9, 10, 17, 18, 25, 26, 33, 34, 41, 42, 65, 66, 129, 130]
    rng = np.random.Generator(np.random.PCG64(rows))
    hit = np.concatenate([(rng.random((rows, 1)) < 0.5) & (rng.random((rows, c)) < 0.5) for c in sizes], axis=1)
    expected, at = {}, 0
    for c in sizes:
        f = hit[:, at : at + c].astype(np.float32)
        pair = np.rint(f.T @ f).astype(np.int64)
        expected.update({frozenset((at + a + 1, at + b + 1)): int(pair[a, b]) for a in range(c) for b in range(a + 1, c)})
        at += c
    off, items = _csr(hit)
    with tf.Database.from_csr(off, items, 0.094) as db:
        got = db.mine(engine="resident", **opts)
        assert got.as_dict() == expected
        assert got.stats["path_supports"][2] > at * at   # more than the top family on the tensor path


# 91 items give 4,095 frequent pairs, 45 items 990; each lone item adds one set.
@pytest.mark.parametrize("wide,lone", [(91, 0), (91, 1), (91, 2), (45, 33), (45, 34), (45, 35), (2, 0)])
def test_result_sort_boundary(oracle_mod, tmp_path, wide, lone):
    rng = np.random.Generator(np.random.PCG64(lone))
    hit = np.zeros((2000 + 900 * lone, wide + lone), dtype=bool)
    hit[:2000, :wide] = rng.random((2000, wide)) < 0.5
    for k in range(lone):
        hit[2000 + 900 * k : 2900 + 900 * k, wide + k] = True
    path = str(tmp_path / "d.txt")
    with open(path, "w") as f:
        f.writelines(" ".join(map(str, np.flatnonzero(r) + 1)) + "\n" for r in hit if r.any())
    minsup = 369.5 / sum(r.any() for r in hit)   # between the supports of pairs and triples
    expected = oracle_mod.mine_file(path, minsup)
    assert len(expected) == wide * (wide - 1) // 2 + lone
    with tf.Database.from_file(path, minsup) as db:
        for engine in ("resident", "batched"):
            assert db.mine(engine=engine).as_dict() == expected


@pytest.mark.parametrize("items", [31, 33, 1023, 1025, 32_768, 32_769])
def test_dense_id_tables(items):
    rng = np.random.Generator(np.random.PCG64(items))
    rows = 300
    held = [np.sort(rng.choice(items, size=min(40, items), replace=False)) + 1 for _ in range(rows)]
    held[7] = np.arange(1, items + 1)   # every item occurs; most supports tie
    off = np.concatenate([[0], np.cumsum([len(h) for h in held])]).astype(np.int64)
    flat = np.concatenate(held).astype(np.int32)
    sup = np.bincount(flat, minlength=items + 1)[1:]
    minc = 2 if items < 2000 else int(np.sort(sup)[-40])
    keep = sup >= minc
    with tf.Database.from_csr(off, flat, (minc - 0.5) / rows) as db:
        assert db.info["n_dense"] == int(keep.sum())
        counts, _ = db.count_wave([[]], 1, counter="lop3")
        assert (counts[0] == sup[keep]).all()
    with tf.Database.from_csr(off, flat, 0.5 / rows) as db:
        counts, _ = db.count_wave([[], [items - 1]], 1, counter="lop3")
        assert db.info["n_dense"] == items and (counts[0] == sup).all()
        assert counts[1][items - 1] == sup[items - 1] and counts[1].sum() == sum(len(h) for h in held if items in h)


def test_mine_with_tied_supports(oracle_mod, tmp_path):
    rng = np.random.Generator(np.random.PCG64(5))
    p = 1.0 / np.arange(1, 2001) ** 0.7
    path = str(tmp_path / "d.txt")
    with open(path, "w") as f:
        for _ in range(3000):
            f.write(" ".join(map(str, np.unique(rng.choice(2000, size=7, p=p / p.sum())))) + "\n")   # id 0 too
    expected = oracle_mod.mine_file(path, 0.0012)
    with tf.Database.from_file(path, 0.0012) as db:
        assert db.info["n_dense"] > 1024
        assert db.mine().as_dict() == expected
