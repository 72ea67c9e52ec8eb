"""Plans batched with extensions of theirs that cannot match: counts, supports
and per-graph counts are those of each plan alone."""
import numpy as np
import pytest

import geneva_b200 as gv

pytestmark = pytest.mark.gpu

GRAPHS = 5

# a plan and, after it, the edges that extend it by a vertex label or an edge
# label that the data lack
BASES = [
    ("v 0 1\nv 1 2\n", "e 0 1 1\n"),                                                     # one edge
    ("v 0 1\nv 1 2\nv 2 3\n", "e 0 1 1\ne 1 2 1\n"),                                     # a path
    ("v 0 1\nv 1 2\nv 2 2\n", "e 0 1 1\ne 0 2 1\n"),                                     # a restriction
    ("v 0 1\nv 1 2\nv 2 3\n", "e 0 1 1\ne 1 2 1\ne 0 2 2\n"),                            # a triangle: a reduction
    ("v 0 1\nv 1 2\nv 2 3\nv 3 2\n", "e 0 1 1\ne 1 2 1\ne 0 2 2\ne 2 3 1\n"),            # and a tail
]


def extended(vertices, edges, at, label, edge_label):
    n = vertices.count("v")
    return vertices + f"v {n} {label}\n" + edges + f"e {at} {n} {edge_label}\n"


@pytest.fixture(scope="module")
def db(native):
    """Per graph g: g + 1 triangles 1 - 2 - 3 (2 and 3 by label 1, 1 and 3 by
    label 2), a second vertex 2 on each 1 and one on each 3; none in the last."""
    labels, edges, first = [0], [], [1]
    for g in range(GRAPHS):
        for _ in range(g + 1 if g + 1 < GRAPHS else 0):
            a = len(labels)
            labels += [1, 2, 3, 2, 2]
            edges += [(a, a + 1, 1), (a + 1, a + 2, 1), (a, a + 2, 2), (a, a + 3, 1), (a + 2, a + 4, 1)]
        labels.append(4)
        first.append(len(labels))
    e = np.array(edges, np.uint32)
    d = gv.Database.from_edges(np.array(labels, np.uint32), e[:, 0], e[:, 1], e[:, 2])
    d.set_graphs(first)
    yield d
    d.close()


@pytest.mark.parametrize("mode", [gv.MODE_DV, gv.MODE_SV])
@pytest.mark.parametrize("base", range(len(BASES)))
@pytest.mark.parametrize("label,edge_label", [(99, 1), (2, 7)])
def test_base_with_a_dead_extension(db, base, mode, label, edge_label):
    vertices, edges = BASES[base]
    n = vertices.count("v")
    texts = [vertices + edges] + [extended(vertices, edges, at, label, edge_label) for at in range(n)]
    want = [gv.batch_count(db, [gv.Plan.from_text(t, mode)], graph_counts=True, support=True, host_rounds=True)[:2]
            for t in texts]
    assert int(want[0][0][0]) > 0 and int(want[0][1][1][0]) == GRAPHS - 1
    for rounds in ({}, {"device_rounds": True}, {"host_rounds": True}):
        plans = gv.Plan.batch_from_texts(texts, mode)
        counts, (per_graph, support), _ = gv.batch_count(db, plans, graph_counts=True, support=True, **rounds)
        for i, (c, (g, s)) in enumerate(want):
            assert int(counts[i]) == int(c[0]), (i, rounds)
            assert int(support[i]) == int(s[0]), (i, rounds)
            assert np.array_equal(per_graph[i], g[0]), (i, rounds)
