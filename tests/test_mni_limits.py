"""MNI searches whose queues run over: rounds with room for a few dozen pieces
give the supports of the CPU oracle, and a run over a graph that fills the
default queues stops soon after it is cancelled."""
import ctypes
import threading
import time

import numpy as np
import pytest

import geneva_b200 as gv
from geneva_b200 import workloads
from test_mni_pieces import hub_graph

pytestmark = pytest.mark.gpu

SQUARE = "v 0 2\nv 1 3\nv 2 3\nv 3 4\ne 0 1 1\ne 0 2 1\ne 1 3 1\ne 2 3 1\n"
LIMITS = [(32, 32, 1), (33, 40, 2), (96, 1 << 18, 512), (1 << 18, 32, 512), (4096, 4096, 1)]


def open_db(labels, edges):
    return gv.Database.from_edges(labels, edges[:, 0], edges[:, 1], np.ones(len(edges), np.uint32))


def patterns_of(labels):
    """Cycles, a tailed triangle and a star over the given vertex labels."""
    a, b, c, d = labels
    v = f"v 0 {a}\nv 1 {b}\nv 2 {c}\nv 3 {d}\n"
    return [v + "e 0 1 1\ne 1 2 1\ne 2 3 1\ne 0 3 1\n",
            v + "e 0 1 1\ne 1 2 1\ne 0 2 1\ne 0 3 1\n",
            v + "e 0 1 1\ne 0 2 1\ne 0 3 1\n",
            v + "e 0 1 1\ne 1 2 1\ne 2 3 1\ne 0 3 1\ne 0 2 1\ne 1 3 1\n"]


@pytest.mark.parametrize("pieces,roots,groups", LIMITS)
def test_hub_pairs(native, pieces, roots, groups):
    """Squares under hubs of 1,500 leaves: every leaf is a root whose lane
    gives up, far more of them than there is room for."""
    labels, edges = hub_graph(1500, 3, 2)
    db = open_db(labels, edges)
    db.set_limits(mni_pieces=pieces, mni_roots=roots, mni_groups=groups)
    texts = [SQUARE, SQUARE.replace("v 3 4\n", "v 3 4\nv 4 1\n") + "e 0 4 1\n"]
    for plain in (False, True):
        for cap, want in ((0, 2), (1, 1)):
            sup, _ = gv.mni_support(db, texts, cap=cap, plain=plain)
            assert [int(x) for x in sup] == [want, want]
    db.close()


@pytest.mark.parametrize("pieces,roots,groups", LIMITS)
@pytest.mark.parametrize("scale,edges,seed", [(9, 4000, 3), (12, 30000, 4)])
def test_rmat_against_oracle(native, oracle, pieces, roots, groups, scale, edges, seed):
    g = workloads.rmat_graph(scale, edges, 2, None, seed=seed, name="limits")
    db = gv.Database.from_edges(g.vlabels, g.src, g.dst, g.elabels)
    db.set_limits(mni_pieces=pieces, mni_roots=roots, mni_groups=groups)
    texts = [t for l in ((1, 1, 1, 1), (1, 2, 1, 2), (2, 2, 1, 1), (1, 1, 2, 1)) for t in patterns_of(l)]
    og = oracle.mni_graph(g.vlabels, g.src, g.dst, g.elabels)
    for cap in (0, 7):
        want = [oracle.mni(og, t, cap=cap)[0] for t in texts]
        for plain in (False, True):
            sup, _ = gv.mni_support(db, texts, cap=cap, plain=plain)
            assert [int(x) for x in sup] == want
    oracle.mni_graph_free(og)
    db.close()


def test_limits_are_checked(native):
    labels, edges = hub_graph(3, 1, 0)
    db = open_db(labels, edges)
    for bad in ({"mni_pieces": 31}, {"mni_roots": 1}):
        with pytest.raises(gv.GenevaError):
            db.set_limits(**bad)
    db.close()


@pytest.mark.parametrize("limits", [{}, {"mni_pieces": 4096, "mni_roots": 4096}])
def test_cancelled_run_returns_soon(native, limits):
    """Two hubs (label 2) of 600,000 leaves (3) with a vertex (4) each, and two
    more vertices 4 that join a leaf of either hub: every part of a square hub -
    leaf - 4 - leaf is there, no square is, and each search tries the pairs of a
    hub's leaves, 3.6e11, a run of minutes.  It is cancelled after a second and
    returns within half a second."""
    n = 600000
    hub = np.array([1, 2], np.uint32).repeat(n)
    leaf = np.arange(3, 3 + 2 * n, dtype=np.uint32)
    join = np.array([3 + 4 * n, 4 + 4 * n], np.uint32)
    labels = np.concatenate([[0, 2, 2], np.full(2 * n, 3), np.full(2 * n, 4), [4, 4]]).astype(np.uint32)
    src = np.concatenate([hub, leaf, leaf[:2], leaf[n:n + 2]])
    dst = np.concatenate([leaf, leaf + 2 * n, join, join])
    db = gv.Database.from_edges(labels, src, dst, np.ones(len(src), np.uint32))
    db.set_limits(**limits)
    cancel, set_at = ctypes.c_int(0), []

    def stop():
        set_at.append(time.perf_counter())
        cancel.value = 1

    timer = threading.Timer(1.0, stop)
    timer.start()
    try:
        with pytest.raises(gv.GenevaError):
            gv.mine(db, 4, 2, support="mni", cancel=cancel)
        late = time.perf_counter() - set_at[0] if set_at else None
    finally:
        timer.cancel()
    assert late is not None and late < 0.5, late
    db.close()
