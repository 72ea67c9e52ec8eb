"""Runs within their budget, and on a device whose free memory lies in the
frontier regions' pool."""
import numpy as np
import pytest
import torch

import geneva_b200 as gv
from geneva_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graphs(native):
    db = workloads.graph_database(300, 10, 30, 3.0, 4, None, 2, seed=77, name="small")
    gdb = gv.Database.from_edges(db.vlabels, db.src, db.dst, db.elabels)
    gdb.set_graphs(db.first)
    plans = [gv.Plan.from_text(p) for p in workloads.sample_patterns(db, 40, 3, 5, seed=3)]
    yield gdb, plans
    gdb.close()


def test_regions_and_schedule_fit_the_budget(graphs):
    """Regions of 1 MiB need more than 2 MiB with their schedule, and no more
    than the budget is taken although runs are rounded up to 256 MiB."""
    gdb, plans = graphs
    gdb.set_tuning(64, 32, round_region_mb=1)
    want, _, stats = gv.batch_count(gdb, plans)
    assert stats["device_rounds"] > 0
    got, _, stats = gv.batch_count(gdb, plans, budget_bytes=2 << 20)
    assert stats["device_rounds"] == 0 and np.array_equal(got, want)
    got, _, stats = gv.batch_count(gdb, plans, budget_bytes=8 << 20)
    assert stats["device_rounds"] > 0 and np.array_equal(got, want)


def test_kept_regions_are_given_back_when_the_device_is_full(graphs):
    """64 GiB of regions stay with their pool after a run; a query's 15 GB
    frontier is then allocated on a device that has 4 GiB free beside them."""
    gdb, plans = graphs
    free, total = torch.cuda.mem_get_info()
    if free < (100 << 30):
        pytest.skip("needs 100 GiB of free device memory")
    leaves = 50_000
    labels = np.array([0, 1] + [2] * leaves, np.uint32)
    leaf = np.arange(2, 2 + leaves, dtype=np.uint32)
    star = gv.Database.from_edges(labels, np.ones(leaves, np.uint32), leaf, np.ones(leaves, np.uint32))
    gdb.set_tuning(64, 32, round_region_mb=32 << 10)
    _, _, stats = gv.batch_count(gdb, plans)
    assert stats["device_rounds"] > 0
    torch.cuda.synchronize()
    kept, _ = torch.cuda.mem_get_info()
    assert kept < total - (64 << 30)  # the pool may have held some of it before
    fill = torch.empty(kept - (4 << 30), dtype=torch.uint8, device="cuda")
    res = gv.match(star, gv.Plan.from_text("v 0 1\nv 1 2\nv 2 2\ne 0 1 1\ne 0 2 1\n"), budget_bytes=40 << 30)
    assert res.num_rows == leaves * (leaves - 1) // 2
    del res, fill
    torch.cuda.empty_cache()
    star.close()
    gdb.set_tuning(64, 32, round_region_mb=2048)
