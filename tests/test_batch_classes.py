"""Rounds whose light class starts while the fused class's launch runs: what it
reads of the round before is the same however the two overlap."""
import numpy as np
import pytest

import geneva_b200 as gv
from geneva_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused,light", [(1, 40), (40, 1), (30, 30)])
def test_repeated_runs_agree(native, fused, light):
    db = workloads.graph_database(2000, 20, 60, 4.0, 3, None, 2, seed=5, name="classes")
    gdb = gv.Database.from_edges(db.vlabels, db.src, db.dst, db.elabels)
    gdb.set_graphs(db.first)
    rng = np.random.default_rng(fused)

    def path(n):
        return "".join(f"v {i} {1 + rng.integers(3)}\n" for i in range(n)) + \
               "".join(f"e {i} {i + 1} {1 + rng.integers(2)}\n" for i in range(n - 1))

    texts = [path(6) + "e 0 2 1\ne 3 5 2\n" for _ in range(fused)] + [path(6) for _ in range(light)]
    plans = [gv.Plan.from_text(t) for t in texts]
    want, want_sup, _ = gv.batch_count(gdb, plans, support=True, host_rounds=True)
    assert int(want.sum()) > 0
    for _ in range(25):
        got, sup, stats = gv.batch_count(gdb, plans, support=True)
        assert stats["device_rounds"] > 0
        assert np.array_equal(got, want) and np.array_equal(sup, want_sup)
    gdb.close()
