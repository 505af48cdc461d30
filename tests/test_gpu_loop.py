"""Device-driven wave loops (csrc/resident.cu: k_res_loop and the graph) that end at their time limit and
are launched again: with `small_pools` every launch ends after one wave.  The search must not
notice."""
import pytest

import tensorfim_b200 as tf
from conftest import golden_input, load_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("name", ["cfg1_full", "cfg1_t03", "cfg5_s002", "cfg3_base_t06"])
def test_loop_continues_where_it_stopped(tmp_path, name, graphs):
    fx = load_golden(name)
    with tf.Database.from_file(golden_input(fx, tmp_path), fx["spec"]["minsup"]) as db:
        for la in (False, "learned"):
            whole = db.mine(engine="resident", lookahead=la, graphs=graphs)
            cut = db.mine(engine="resident", lookahead=la, graphs=graphs, small_pools=True)
            assert cut.as_dict() == whole.as_dict() == fx["expected"]
            if not la:   # every family is counted once, in whatever waves
                assert cut.stats["supports"] == whole.stats["supports"] and cut.stats["nodes"] == whole.stats["nodes"]
            if not graphs:
                assert cut.stats["launches"] >= cut.stats["waves"] > 1
                if name.startswith("cfg1"):   # all waves are the loop's
                    assert whole.stats["launches"] < whole.stats["waves"] + 4
