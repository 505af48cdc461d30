"""Families moved to universes of their own (csrc/resident.cu, projection): the mined sets are the
reference's whatever the number of transactions, so whatever the compressed rows' boundaries.
`small_pools` projects at any length; without it only databases of at least 2^17 transactions do."""
import numpy as np
import pytest

import tensorfim_b200 as tf
from tensorfim_b200 import synth

from conftest import load_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [dict(lookahead="learned"), dict(lookahead="filtered", graphs=True),
                                  dict(lookahead="all", superset=True), dict(lookahead=False, counter="lop3"),
                                  dict(lookahead="filtered", counter="tensor"), dict(counter="i8", wave_cap=500),
                                  dict(lookahead="learned", small_pools=True)])
def test_long_database_matches_reference(opts):
    reps = 3   # 147,000 transactions
    fx = load_golden("cfg3_base_t06")
    db0 = synth.generate(3, replicas=reps)
    with tf.Database.from_csr(db0.offsets, db0.items, 0.06) as db:
        assert db.info["words_per_row"] >= 4096
        got = db.mine(engine="resident", **opts).as_dict()
    assert got == {k: v * reps for k, v in fx["expected"].items()}


@pytest.mark.parametrize("rows", [33, 64, 2047, 2049, 32_767, 32_769, 100_003])
def test_compressed_row_boundaries(oracle_mod, tmp_path, rows):
    rng = np.random.Generator(np.random.PCG64(rows))
    probs = [rng.dirichlet(np.full(4, 0.6)) for _ in range(12)]
    db0 = synth.categorical(rows, probs, rng)
    path = str(tmp_path / "d.txt")
    synth.write_fimi(path, db0)
    expected = oracle_mod.mine_file(path, 0.07)
    with tf.Database.from_csr(db0.offsets, db0.items, 0.07) as db:
        for graphs in (False, True):
            assert db.mine(engine="resident", small_pools=True, graphs=graphs).as_dict() == expected


# 420 items: positions in 14 groups of 32, two chunks of groups.  Three wide clusters are compressed
# through transposed transactions, forty narrow ones word by word; runs of a cluster's transactions leave
# tiles without any and last words that end many tiles later.
@pytest.mark.parametrize("clusters,prob,minsup", [(3, 0.5, 0.06), (40, 0.8, 0.014)])
@pytest.mark.parametrize("runs", [1, 700, 4001, 20_011])
def test_groups_of_items(oracle_mod, tmp_path, clusters, prob, minsup, runs):
    rows, per = 20_011, 420 // clusters
    rng = np.random.Generator(np.random.PCG64(clusters + runs))
    cluster = np.arange(rows) // runs % clusters if runs < rows else np.arange(rows) * clusters // rows
    own = np.arange(clusters * per) % clusters == cluster[:, None]
    hit = own & (rng.random(own.shape) < prob)
    path = str(tmp_path / "d.txt")
    with open(path, "w") as f:
        f.writelines(" ".join(map(str, np.flatnonzero(r) + 1)) + "\n" for r in hit if r.any())
    expected = oracle_mod.mine_file(path, minsup)
    with tf.Database.from_file(path, minsup) as db:
        assert db.mine(engine="resident", small_pools=True).as_dict() == expected
