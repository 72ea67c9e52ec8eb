"""Budgets that split tasks or make them wait: a plan that ends where others go
on counts the rows of such a task once."""
import numpy as np
import pytest

import geneva_b200 as gv
from geneva_b200 import workloads

pytestmark = pytest.mark.gpu

PATH = "v 0 1\nv 1 1\nv 2 1\nv 3 1\n"
NESTED = ["v 0 1\nv 1 1\ne 0 1 1\n",
          "v 0 1\nv 1 1\nv 2 1\ne 0 1 1\ne 1 2 1\n",
          "v 0 1\nv 1 1\nv 2 1\ne 0 1 1\ne 0 2 1\n",
          "v 0 1\nv 1 1\nv 2 1\ne 0 1 1\ne 1 2 1\ne 0 2 1\n",
          PATH + "e 0 1 1\ne 1 2 1\ne 2 3 1\n",
          PATH + "e 0 1 1\ne 0 2 1\ne 0 3 1\n",
          PATH + "e 0 1 1\ne 1 2 1\ne 0 2 1\ne 0 3 1\n"]


@pytest.fixture(scope="module")
def db(native):
    d = workloads.graph_database(200, 10, 30, 3.0, 1, None, 1, seed=5, name="budget")
    gdb = gv.Database.from_edges(d.vlabels, d.src, d.dst, d.elabels)
    gdb.set_graphs(d.first)
    yield gdb
    gdb.close()


@pytest.mark.parametrize("mode", [gv.MODE_DV, gv.MODE_SV])
@pytest.mark.parametrize("budget", [2048, 16 << 10, 100 << 10])
def test_nested_plans(db, budget, mode):
    """Each plan counted alone: its own steps write, only its last one counts."""
    want = [gv.batch_count(db, [gv.Plan.from_text(t, mode)], graph_counts=True, support=True)[:2] for t in NESTED]
    plans = gv.Plan.batch_from_texts(NESTED, mode)
    rounds = gv.batch_count(db, plans, host_rounds=True)[2]["rounds"]
    counts, (per_graph, support), stats = gv.batch_count(db, plans, graph_counts=True, support=True, budget_bytes=budget)
    assert stats["rounds"] > rounds  # some task came back
    for i, (c, (g, s)) in enumerate(want):
        assert int(counts[i]) == int(c[0]) > 0, i
        assert int(support[i]) == int(s[0]), i
        assert np.array_equal(per_graph[i], g[0]), i
