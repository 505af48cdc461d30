"""The resident engine's wave pack (csrc/resident.cu, res_pack) when a wave's packed tensor-core jobs
are so little work that they move to the CUDA cores: the whole block has to take that decision
alike, in the host-driven, the graph-driven and the device-driven wave loop."""
import os
import re

import numpy as np
import pytest

import tensorfim_b200 as tf
from tensorfim_b200 import _lib, synth

CSRC = os.path.join(os.path.dirname(os.path.abspath(tf.__file__)), "csrc")


def test_wave_sums_are_only_read_after_the_decision():
    """Every thread reads the wave's shared sums to decide, with no barrier behind the reads, so
    nothing may store to them from there on."""
    with open(os.path.join(CSRC, "resident.cu")) as f:
        src = f.read()
    body = src[src.index("void res_pack("):src.index("void publish_status(")]
    after = body[body.index("const bool few_pk"):]
    for name in ("s_words", "s_cost", "s_pk_work", "s_pk_cost"):
        assert not re.search(name + r"(\[\d\])?\s*[-+]?=(?!=)", after), name
        assert not re.search(r"atomic\w+\(\s*\(?[^,;]*&\s*" + name, after), name


@pytest.mark.gpu
@pytest.mark.parametrize("opts", [dict(superset=True), dict(graphs=True), dict()])
def test_little_packed_work(oracle_mod, tmp_path, opts):
    """26 items of 40,003 transactions (1,280 words a row): waves of tens of families with 8 to 24
    tail rows, well below the packed tiles' least work."""
    rng = np.random.Generator(np.random.PCG64(8))
    hit = rng.random((40_003, 26)) < rng.uniform(0.5, 0.8, 26)
    off = np.concatenate([[0], np.cumsum(hit.sum(1))]).astype(np.int64)
    items = (np.nonzero(hit)[1] + 1).astype(np.int32)
    path = str(tmp_path / "d.txt")
    synth.write_fimi(path, synth.Database(offsets=off, items=items, n_items=26))
    expected = oracle_mod.mine_file(path, 0.15)
    tc = _lib.PATHS.index("tc")
    with tf.Database.from_csr(off, items, 0.15) as db:
        # asked for, the packed tiles take these families; left to the automatic choice only the first one does
        wide = db.mine(engine="resident", counter="i8", lookahead=False, **opts)
        assert wide.as_dict() == expected and wide.stats["path_supports"][tc] > 26 * 26
        first = db.mine(engine="resident", lookahead=False, **opts)
        assert first.as_dict() == expected and first.stats["path_supports"][tc] <= 26 * 26
        for _ in range(200):
            r = db.mine(engine="resident", lookahead=False, **opts)
            assert (r.items == first.items).all() and (r.offsets == first.offsets).all()
            assert (r.supports == first.supports).all()
            if "superset" not in opts:   # (what that check prunes depends on the order in which sets are found)
                assert r.stats["supports"] == first.stats["supports"]
