"""Batched rounds in one pass: pages at the edges of their sizes, on graphs
whose counts have a closed form."""
from math import comb

import numpy as np
import pytest

import geneva_b200 as gv

pytestmark = pytest.mark.gpu


def stars(n, hubs):
    """`hubs` hubs (label 1) with n leaves (label 2) each; every leaf has one
    vertex (label 3) of its own."""
    labels, edges = [0], []
    for _ in range(hubs):
        labels.append(1)
        hub = len(labels) - 1
        for _ in range(n):
            labels += [2, 3]
            edges += [(hub, len(labels) - 2), (len(labels) - 2, len(labels) - 1)]
    return np.array(labels, np.uint32), np.array(edges, np.uint32)


def star_patterns(n, hubs):
    """(query text, embeddings): stars of up to three leaves, then with a tail
    on one leaf and on two, and a triangle that no star has."""
    v = {1: "v 0 1\n", 2: "v 0 1\nv 1 2\n", 3: "v 0 1\nv 1 2\nv 2 2\n", 4: "v 0 1\nv 1 2\nv 2 2\nv 3 2\n"}
    return [
        (v[2] + "e 0 1 1\n", hubs * n),
        (v[3] + "e 0 1 1\ne 0 2 1\n", hubs * comb(n, 2)),
        (v[4] + "e 0 1 1\ne 0 2 1\ne 0 3 1\n", hubs * comb(n, 3)),
        (v[3] + "v 3 3\ne 0 1 1\ne 0 2 1\ne 1 3 1\n", hubs * n * (n - 1)),
        (v[4] + "v 4 3\ne 0 1 1\ne 0 2 1\ne 0 3 1\ne 1 4 1\n", hubs * n * comb(n - 1, 2)),
        (v[3] + "v 3 3\nv 4 3\ne 0 1 1\ne 0 2 1\ne 1 3 1\ne 2 4 1\n", hubs * comb(n, 2)),
        (v[3] + "e 0 1 1\ne 0 2 1\ne 1 2 1\n", 0),
    ]


@pytest.mark.parametrize("rows_per_item", [32, 64, 128])
@pytest.mark.parametrize("n,hubs", [(1, 1), (2, 33), (8, 4), (31, 3), (32, 2), (33, 1), (64, 5), (127, 1), (129, 2)])
def test_star_counts(native, n, hubs, rows_per_item):
    labels, edges = stars(n, hubs)
    db = gv.Database.from_edges(labels, edges[:, 0], edges[:, 1], np.ones(len(edges), np.uint32))
    db.set_graphs([1 + i * (1 + 2 * n) for i in range(hubs + 1)])
    db.set_tuning(rows_per_item, 32)
    texts, want = zip(*star_patterns(n, hubs))
    for mode in (gv.MODE_DV, gv.MODE_SV):
        plans = gv.Plan.batch_from_texts(list(texts), mode)
        counts, (per_graph, support), st = gv.batch_count(db, plans, graph_counts=True, support=True)
        assert st["device_rounds"] == st["rounds"] > 0
        assert [int(c) for c in counts] == list(want)
        assert [int(s) for s in support] == [hubs if w else 0 for w in want]
        for row, w in zip(per_graph, want):
            assert (row == w // hubs).all()
    db.close()


def test_stepped_halves(native):
    """Runs in two halves, whose rounds the host launches one at a time."""
    labels, edges = stars(40, 3)
    db = gv.Database.from_edges(labels, edges[:, 0], edges[:, 1], np.ones(len(edges), np.uint32))
    texts, want = zip(*star_patterns(40, 3))
    reps = 12288 // len(texts) + 1
    plans = gv.Plan.batch_from_texts(list(texts) * reps)
    counts, _, st = gv.batch_count(db, plans)
    assert st["device_rounds"] == 0 and st["rounds"] > 0
    assert [int(c) for c in counts] == list(want) * reps
    db.close()


@pytest.mark.parametrize("m", [7, 12, 13, 16])
def test_wide_rows(native, m):
    """Rows wide enough for pages of 64 and 32 rows: paths of m vertices along
    one long path whose labels repeat 1, 2, 3."""
    n = 3 * 500
    labels = np.array([0] + [1 + i % 3 for i in range(n)], np.uint32)
    a = np.arange(1, n, dtype=np.uint32)
    db = gv.Database.from_edges(labels, a, a + 1, np.ones(n - 1, np.uint32))
    texts = ["".join(f"v {i} {1 + (i + s) % 3}\n" for i in range(m)) + "".join(f"e {i} {i + 1} 1\n" for i in range(m - 1))
             for s in range(3)]
    counts, _, st = gv.batch_count(db, gv.Plan.batch_from_texts(texts))
    assert st["device_rounds"] > 0
    assert [int(c) for c in counts] == [len(range(s, n - m + 1, 3)) for s in range(3)]
    db.close()


@pytest.mark.parametrize("hubs,n", [(1, 300), (3, 2100), (2, 4097)])
def test_long_lists(native, hubs, n):
    """Lists cut into pieces: hubs joined in a path, their leaves paired, so
    that extensions with and without fused checks walk thousands of
    candidates per row."""
    labels, edges, first = [0], [], []
    for h in range(hubs):
        labels.append(1)
        hub = len(labels) - 1
        first.append(hub)
        leaf = list(range(len(labels), len(labels) + n))
        labels += [2] * n
        edges += [(hub, v) for v in leaf] + [(leaf[i], leaf[i + 1]) for i in range(0, n - 1, 2)]
        if h:
            edges.append((first[-2], hub))
    e = np.array(edges, np.uint32)
    db = gv.Database.from_edges(np.array(labels, np.uint32), e[:, 0], e[:, 1], np.ones(len(e), np.uint32))
    pairs = n // 2
    texts = ["v 0 1\nv 1 2\nv 2 2\ne 0 1 1\ne 0 2 1\ne 1 2 1\n",              # triangles
             "v 0 1\nv 1 2\nv 2 2\ne 0 1 1\ne 0 2 1\n",                       # two leaves of a hub
             "v 0 2\nv 1 1\nv 2 1\nv 3 2\ne 0 1 1\ne 1 2 1\ne 2 3 1\n",       # leaf, hub, hub, leaf
             "v 0 1\nv 1 2\nv 2 2\nv 3 2\ne 0 1 1\ne 0 2 1\ne 1 2 1\ne 0 3 1\n"]  # triangle and a leaf
    want = [hubs * pairs, hubs * n * (n - 1) // 2, (hubs - 1) * n * n, hubs * pairs * (n - 2)]
    for R in (32, 64):
        db.set_tuning(R, 32)
        counts, _, st = gv.batch_count(db, gv.Plan.batch_from_texts(texts))
        assert st["device_rounds"] > 0
        assert [int(c) for c in counts] == want
    db.close()
