"""The launch shape of counted rounds: what the tuner keeps was timed on them,
and every shape gives the oracle's counts there."""
import numpy as np
import pytest

import geneva_b200 as gv
from geneva_b200 import workloads

pytestmark = pytest.mark.gpu


def test_tuner_shares_long_lists(native):
    """Under a hub of 200,000 leaves one lane walking the list alone takes many
    times what a warp takes, so the tuner may not choose to never share it."""
    n = 200_000
    labels = np.full(n + 2, 2, dtype=np.uint32)
    labels[1] = 1
    leaf = np.arange(2, n + 2, dtype=np.uint32)
    src = np.concatenate([np.ones(n, np.uint32), leaf[:-1]])
    dst = np.concatenate([leaf, leaf[1:]])
    db = gv.Database.from_edges(labels, src, dst, np.ones(len(src), np.uint32))
    plans = [gv.Plan.from_text(t) for t in ("v 0 1\nv 1 2\nv 2 2\ne 0 1 1\ne 1 2 1\n",
                                            "v 0 1\nv 1 2\nv 2 2\ne 0 1 1\ne 1 2 1\ne 0 2 1\n")]
    for _ in range(8):
        t = db.autotune(plans)
        assert t["hub"] <= 64 and db.tuning["hub"] == t["hub"]
        assert t["shapes_tried"] == 12 and 0 < t["ms"] <= t["default_ms"]
    db.close()


@pytest.mark.parametrize("rows_per_item,hub", [(32, 0), (64, 0), (128, 1), (64, 1 << 30), (32, 5), (128, 32)])
def test_shapes_of_counted_rounds(native, oracle, rows_per_item, hub):
    """Hub 0 sends every row's candidates through the warp-shared path of the
    counted kernels, 1 << 30 none; one-pass rounds have no such path."""
    db = workloads.graph_database(300, 10, 30, 3.0, 4, None, 2, seed=77, name="small")
    gdb = gv.Database.from_edges(db.vlabels, db.src, db.dst, db.elabels)
    gdb.set_graphs(db.first)
    og = oracle.from_edges(db.vlabels, db.src, db.dst, db.elabels)
    pats = [p for p in workloads.sample_patterns(db, 60, 3, 6, seed=22) if oracle.count(og, p, cap_rows=1_000_000) is not None]
    want_counts, want_sup, want_gc = oracle.many_graph_counts(og, pats, db.first)
    gdb.set_tuning(rows_per_item, hub)
    plans = [gv.Plan.from_text(p) for p in pats]
    for host_rounds in (True, False):
        counts, (gc, sup), stats = gv.batch_count(gdb, plans, graph_counts=True, support=True, host_rounds=host_rounds)
        assert (stats["device_rounds"] == 0) == host_rounds
        assert np.array_equal(counts, want_counts) and np.array_equal(sup, want_sup)
        assert all(np.array_equal(gc[i], want_gc[i]) for i in range(len(pats)))
    oracle.free(og)
    gdb.close()
