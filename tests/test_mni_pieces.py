"""MNI searches that outlast a warp's budget and are cut into pieces
(mni_piece_kernel): hubs whose neighbour pairs must nearly all be tried."""
import numpy as np
import pytest

import geneva_b200 as gv


def hub_graph(leaves, hubs, closed):
    """`hubs` hubs (label 2), each with one root (1) and `leaves` leaves (3);
    every leaf has a vertex (4) of its own, and in the first `closed` hubs the
    last two leaves share one more."""
    labels, edges = [0], []

    def vertex(label):
        labels.append(label)
        return len(labels) - 1

    for h in range(hubs):
        hub = vertex(2)
        edges.append((vertex(1), hub))
        leaf = [vertex(3) for _ in range(leaves)]
        edges += [(hub, v) for v in leaf] + [(v, vertex(4)) for v in leaf]
        if h < closed:
            d = vertex(4)
            edges += [(leaf[-2], d), (leaf[-1], d)]
    return np.array(labels, np.uint32), np.array(edges, np.uint32)


@pytest.mark.gpu
@pytest.mark.parametrize("leaves,hubs,closed", [(3, 5, 2), (31, 3, 1), (33, 3, 3), (257, 4, 2), (1500, 3, 0), (1500, 3, 2)])
@pytest.mark.parametrize("pendant", [False, True])
def test_hub_pairs(native, leaves, hubs, closed, pendant):
    """A square hub - leaf - vertex - leaf, with the hub's root as a pendant:
    its images lie in the closed hubs only, one hub, two leaves, one vertex
    (and one root) in each."""
    labels, edges = hub_graph(leaves, hubs, closed)
    db = gv.Database.from_edges(labels, edges[:, 0], edges[:, 1], np.ones(len(edges), np.uint32))
    text = "v 0 2\nv 1 3\nv 2 3\nv 3 4\ne 0 1 1\ne 0 2 1\ne 1 3 1\ne 2 3 1\n"
    if pendant:
        text = text.replace("v 3 4\n", "v 3 4\nv 4 1\n") + "e 0 4 1\n"
    for plain in (False, True):
        for cap in (0, 1):
            sup, _ = gv.mni_support(db, [text, text], cap=cap, plain=plain)
            want = closed if cap == 0 else min(closed, cap)
            assert [int(x) for x in sup] == [want, want]
    db.close()
