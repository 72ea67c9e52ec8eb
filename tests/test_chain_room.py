"""Queries whose frontiers would outgrow a chain's room, and those whose results
outgrow the small buffer: one way through their steps, the oracle's rows."""
import numpy as np
import pytest

import geneva_b200 as gv
from test_match_chunks import small_graphs

pytestmark = pytest.mark.gpu

QUERIES = [
    "v 0 1\nv 1 1\nv 2 1\nv 3 1\ne 0 1 1\ne 1 2 1\ne 2 3 1\n",
    "v 0 1\nv 1 1\nv 2 1\ne 0 1 1\ne 1 2 1\n",
    "v 0 1\nv 1 1\nv 2 1\nv 3 1\ne 0 1 1\ne 0 2 1\ne 0 3 1\n",
    "v 0 1\nv 1 1\nv 2 1\nv 3 1\ne 0 1 1\ne 1 2 1\ne 2 3 1\ne 0 3 1\n",
    "v 0 1\nv 1 1\nv 2 1\nv 3 1\ne 0 1 1\ne 1 2 1\ne 0 2 1\ne 2 3 2\n",
]


@pytest.mark.parametrize("copies,extra,labels", [(400, 4, 1), (400, 6, 3), (3000, 8, 2), (1500, 130, 1), (3000, 130, 2)])
def test_no_step_runs_twice(native, oracle, copies, extra, labels):
    """Counted one by one, a step has a count, a scan and, but for the last of
    a counted query, a write; in a chain it has one launch."""
    lab, src, dst, el = small_graphs(copies, extra, copies + extra)
    lab[1:] = 1 + lab[1:] % labels
    db = gv.Database.from_edges(lab, src, dst, el)
    og = oracle.from_edges(lab, src, dst, el)
    for text in QUERIES:
        want, phases = oracle.match(og, text)
        plan = gv.Plan.from_text(text)
        for count_only in (True, False):
            n0 = gv.kernel_launches()
            res = gv.match(db, plan, count_only=count_only)
            n1 = gv.kernel_launches()
            one_by_one = gv.match(db, plan, count_only=count_only, profile=True)
            n2 = gv.kernel_launches()
            assert res.num_rows == one_by_one.num_rows == len(want)
            assert res.phase_rows == one_by_one.phase_rows == phases, text
            if not count_only:
                assert np.array_equal(res.rows(), want[np.lexsort(want.T[::-1])]), text
            if len(want):
                steps = (n2 - n1 + count_only) // 3
                assert n1 - n0 in (steps, n2 - n1), text
    oracle.free(og)
    db.close()
