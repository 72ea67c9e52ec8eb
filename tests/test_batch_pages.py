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
