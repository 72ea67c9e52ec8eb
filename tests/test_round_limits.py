"""Fallbacks of one-pass rounds and chained steps, with capacities small enough
to reach them: pieces of long lists without room, groups whose lists are walked
one at a time, chains whose tiles stop waiting for one another."""
import numpy as np
import pytest

import geneva_b200 as gv
from geneva_b200 import workloads
from test_match_chunks import CHAIN_QUERIES, small_graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pieces", [1, 33, 1 << 20])
@pytest.mark.parametrize("most", [1, 300, 1 << 26])
def test_long_lists(native, oracle, pieces, most):
    g = workloads.rmat_graph(12, 60000, 3, None, seed=9, name="limits")
    db = gv.Database.from_edges(g.vlabels, g.src, g.dst, g.elabels)
    db.set_limits(round_pieces=pieces, round_sum=most)
    og = oracle.from_edges(g.vlabels, g.src, g.dst, g.elabels)
    texts = []
    for a in (1, 2, 3):
        for b in (1, 2, 3):
            v = f"v 0 {a}\nv 1 {b}\nv 2 {1 + a % 3}\n"
            texts.append(v + "e 0 1 1\ne 1 2 1\n")
            texts.append(v + "e 0 1 1\ne 1 2 1\ne 0 2 1\n")
            if a == b:
                texts.append(v + "v 3 2\ne 0 1 1\ne 1 2 1\ne 0 2 1\ne 2 3 1\ne 0 3 1\n")
    want = [oracle.count(og, t) for t in texts]
    counts, _, stats = gv.batch_count(db, [gv.Plan.from_text(t) for t in texts])
    assert stats["device_rounds"] > 0
    assert counts.tolist() == want and sum(want) > 0
    oracle.free(og)
    db.close()


@pytest.mark.parametrize("polls", [1, 3])
def test_chain_that_gives_up(native, oracle, polls):
    labels, src, dst, el = small_graphs(700, 6, 12)
    db = gv.Database.from_edges(labels, src, dst, el)
    db.set_limits(chain_polls=polls)
    og = oracle.from_edges(labels, src, dst, el)
    for text in CHAIN_QUERIES:
        want, phases = oracle.match(og, text)
        plan = gv.Plan.from_text(text)
        res = gv.match(db, plan)
        assert res.phase_rows == phases, text
        assert np.array_equal(res.rows(), want[np.lexsort(want.T[::-1])]), text
        assert gv.match(db, plan, count_only=True).num_rows == len(want)
    oracle.free(og)
    db.close()


@pytest.fixture(scope="module")
def one_label(native):
    labels, src, dst, el = small_graphs(3000, 6, 3)
    labels[1:] = 1
    db = gv.Database.from_edges(labels, src, dst, el)
    yield db
    db.close()


@pytest.mark.parametrize("polls", [1, 2, 4, 8, 16, 64])
def test_last_step_that_gives_up(one_label, polls):
    """A result beyond the small buffer: the last step runs a second time, and
    its tiles may give up waiting in either run, or in neither."""
    plan = gv.Plan.from_text("v 0 1\nv 1 1\ne 0 1 1\n")
    want = gv.match(one_label, plan, profile=True)
    rows = want.rows()
    assert 256 << 10 < rows.nbytes < 512 << 10
    one_label.set_limits(chain_polls=polls)
    for _ in range(60):
        res = gv.match(one_label, plan)
        assert res.phase_rows == want.phase_rows
        assert np.array_equal(res.rows(), rows)


def test_limits_are_checked(native):
    db = gv.Database.from_edges(np.array([0, 1, 1], np.uint32), np.array([1], np.uint32), np.array([2], np.uint32),
                                np.array([1], np.uint32))
    for limits in ({"round_pieces": (1 << 20) + 1}, {"round_sum": (1 << 26) + 1}):
        with pytest.raises(gv.GenevaError):
            db.set_limits(**limits)
    db.close()
