"""Batched rounds with fewer items than warps, a few per warp, and many: counts and
supports against the counted rounds."""
import numpy as np
import pytest

import geneva_b200 as gv


@pytest.mark.gpu
@pytest.mark.parametrize("vertices", [20000, 100001, 300001])
def test_rounds_of_every_size(native, vertices):
    rng = np.random.default_rng(vertices)
    lab = np.ones(vertices + 1, dtype=np.uint32)
    lab[1:] = 1 + rng.integers(0, 2, vertices)
    a = np.arange(1, vertices, dtype=np.uint32)
    src = np.concatenate([a, a[:-2][rng.random(vertices - 3) < 0.3]])
    dst = src + np.concatenate([np.ones(vertices - 1, np.uint32), np.full(len(src) - vertices + 1, 2, np.uint32)])
    db = gv.Database.from_edges(lab, src, dst, 1 + rng.integers(0, 6, len(src)).astype(np.uint32))
    db.set_graphs(np.append(np.arange(1, vertices + 1, 500), vertices + 1))
    texts = []
    for x in range(1, 7):
        for y in range(1, 7):
            p, q, r = 1 + (x + y) % 2, 1 + x % 2, 1 + y % 2
            texts.append(f"v 0 {p}\nv 1 {q}\nv 2 {r}\ne 0 1 {x}\ne 1 2 {y}\n")
            texts.append(f"v 0 {p}\nv 1 {q}\nv 2 {r}\nv 3 1\ne 0 1 {x}\ne 1 2 {y}\ne 0 2 {x}\ne 2 3 {y}\n")
    plans = [gv.Plan.from_text(t) for t in texts]
    got, support, _ = gv.batch_count(db, plans, support=True)
    want, want_support, _ = gv.batch_count(db, plans, support=True, host_rounds=True)
    assert int(np.sum(want)) > 0
    assert np.array_equal(got, want) and np.array_equal(support, want_support)
    db.close()
