"""gva_match on lists far longer than a CTA's share of an extension's output:
rows, their order and the phase counts against the oracle."""
import numpy as np
import pytest

import geneva_b200 as gv

pytestmark = pytest.mark.gpu


def hub_graph(leaves, hubs, seed):
    """Hubs (label 1) joined to all of their own `leaves` leaves (labels 2 and
    3), random edges among leaves of neighbouring hubs, hubs in a path."""
    rng = np.random.default_rng(seed)
    n = hubs * (1 + leaves)
    labels = np.zeros(n + 1, np.uint32)
    labels[1:] = rng.integers(2, 4, n)
    edges = set()
    hub_ids = [1 + h * (1 + leaves) for h in range(hubs)]
    for h, hub in enumerate(hub_ids):
        labels[hub] = 1
        edges |= {(hub, hub + 1 + i) for i in range(leaves)}
        if h:
            edges.add((hub_ids[h - 1], hub))
    while len(edges) < n + 2 * leaves:
        a, b = sorted(int(x) for x in rng.integers(1, n + 1, 2))
        if a != b and labels[a] != 1 and labels[b] != 1:
            edges.add((a, b))
    e = np.array(sorted(edges), np.uint32)
    return labels, e[:, 0], e[:, 1], np.ones(len(e), np.uint32)


QUERIES = [
    "v 0 1\nv 1 2\nv 2 3\ne 0 1 1\ne 0 2 1\n",                               # no reduction
    "v 0 1\nv 1 2\nv 2 3\ne 0 1 1\ne 0 2 1\ne 1 2 1\n",                       # a triangle
    "v 0 1\nv 1 2\nv 2 2\ne 0 1 1\ne 0 2 1\ne 1 2 1\n",                       # with a restriction
    "v 0 1\nv 1 2\nv 2 3\nv 3 3\ne 0 1 1\ne 0 2 1\ne 1 2 1\ne 0 3 1\n",       # and a tail
    "v 0 1\nv 1 2\nv 2 3\nv 3 2\ne 0 1 1\ne 1 2 1\ne 2 3 1\ne 0 3 1\n",       # a square
    "v 0 1\nv 1 1\nv 2 2\ne 0 1 1\ne 0 2 1\n",
]


@pytest.mark.parametrize("leaves,hubs", [(3, 2), (255, 1), (1300, 2), (5000, 1)])
def test_rows_against_oracle(native, oracle, leaves, hubs):
    labels, src, dst, el = hub_graph(leaves, hubs, leaves)
    db = gv.Database.from_edges(labels, src, dst, el)
    og = oracle.from_edges(labels, src, dst, el)
    for text in QUERIES:
        want, phases = oracle.match(og, text)
        for mode in (gv.MODE_DV, gv.MODE_SV):
            plan = gv.Plan.from_text(text, mode)
            res = gv.match(db, plan)
            rows = res.rows()
            if mode == gv.MODE_DV:
                assert res.phase_rows == phases, text
            # every step takes its rows in order and their candidates ascending
            assert np.array_equal(rows, want[np.lexsort(want.T[::-1])]), text
            counted = gv.match(db, plan, count_only=True)
            assert counted.num_rows == len(want) and counted.phase_rows == res.phase_rows
    oracle.free(og)
    db.close()


def test_budget_still_refuses_the_extension(native):
    """An extension whose rows exceed the budget is refused although the
    reduction after it means that they are never written."""
    labels, src, dst, el = hub_graph(1300, 2, 7)
    db = gv.Database.from_edges(labels, src, dst, el)
    plan = gv.Plan.from_text(QUERIES[1])
    res = gv.match(db, plan)
    assert res.num_rows > 0
    kept = 12 * res.num_rows
    with pytest.raises(gv.GenevaError):
        gv.match(db, plan, budget_bytes=2 * kept)
    db.close()


def small_graphs(copies, extra, seed):
    """`copies` graphs of 24 vertices (labels 1..3, two edge labels), each a
    cycle and `extra` chords."""
    rng = np.random.default_rng(seed)
    labels, edges = [0], set()
    for c in range(copies):
        v0 = len(labels)
        labels += rng.integers(1, 4, 24).tolist()
        edges |= {(v0 + i, v0 + (i + 1) % 24) for i in range(24)}
        while len(edges) < (c + 1) * (24 + extra):
            a, b = sorted(int(x) for x in rng.integers(v0, v0 + 24, 2))
            if a != b and (a, b) not in edges and (b, a) not in edges:
                edges.add((a, b))
    e = np.array(sorted(edges), np.uint32)
    return np.array(labels, np.uint32), e[:, 0], e[:, 1], rng.integers(1, 3, len(e)).astype(np.uint32)


CHAIN_QUERIES = QUERIES + [
    "v 0 1\nv 1 2\ne 0 1 1\n",
    "v 0 1\nv 1 1\nv 2 1\nv 3 1\nv 4 1\ne 0 1 1\ne 1 2 2\ne 2 3 1\ne 3 4 2\n",
    "v 0 1\nv 1 2\nv 2 1\nv 3 2\nv 4 3\ne 0 1 1\ne 1 2 1\ne 2 3 2\ne 0 3 1\ne 3 4 1\n",
    "v 0 2\nv 1 9\ne 0 1 1\n",   # a label that the data lack
    "v 0 2\nv 1 2\nv 2 2\nv 3 2\ne 0 1 2\ne 1 2 2\ne 2 3 2\ne 0 3 2\ne 0 2 2\ne 1 3 2\n",  # likely none
]


# extra chords: 4 keeps frontiers small; 130 makes them outgrow the chain's
# room (dense graphs: degree about 13) and its result buffer
@pytest.mark.parametrize("copies,extra", [(1, 0), (11, 4), (32, 4), (700, 6), (40, 130), (1500, 130)])
def test_chain_against_oracle(native, oracle, copies, extra):
    """Queries on graphs without long lists, whose steps run as a chain: one
    tile, several, as many as there are seeds, outputs without room."""
    labels, src, dst, el = small_graphs(copies, extra, copies + extra)
    db = gv.Database.from_edges(labels, src, dst, el)
    og = oracle.from_edges(labels, src, dst, el)
    for text in CHAIN_QUERIES:
        want, phases = oracle.match(og, text)
        plan = gv.Plan.from_text(text)
        res = gv.match(db, plan)
        assert res.phase_rows == phases, text
        rows = res.rows()
        assert np.array_equal(rows, want[np.lexsort(want.T[::-1])]), text
        counted = gv.match(db, plan, count_only=True)
        assert counted.num_rows == len(want) and counted.phase_rows == phases, text
        # the same rows as the steps that are counted one by one
        assert np.array_equal(gv.match(db, plan, profile=True).rows(), rows), text
    oracle.free(og)
    db.close()


@pytest.mark.parametrize("leaves", [900, 1183, 1184, 2100])
def test_large_read_back(native, leaves):
    """Rows read back in pieces (from 8 MiB on; 1,184 leaves give the first
    such size) equal the closed form, whole and from any row on."""
    labels = np.array([0, 1] + [2] * leaves, np.uint32)
    leaf = np.arange(2, 2 + leaves, dtype=np.uint32)
    db = gv.Database.from_edges(labels, np.ones(leaves, np.uint32), leaf, np.ones(leaves, np.uint32))
    res = gv.match(db, gv.Plan.from_text("v 0 1\nv 1 2\nv 2 2\ne 0 1 1\ne 0 2 1\n"))
    rows = res.rows()
    assert len(rows) == leaves * (leaves - 1) // 2
    i, j = np.tril_indices(leaves, -1)
    pairs = np.sort(rows[:, 1:], axis=1) if (rows[:, 0] == 1).all() else None
    assert pairs is not None
    want = np.stack([leaf[j], leaf[i]], axis=1)
    assert np.array_equal(pairs[np.lexsort(pairs.T[::-1])], want[np.lexsort(want.T[::-1])])
    for first, count in ((0, 1), (1, len(rows) - 1), (len(rows) // 3, len(rows) // 2)):
        assert np.array_equal(res.rows(first, count), rows[first:first + count])
    db.close()
