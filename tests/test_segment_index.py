"""Packed segment records: every label's segment, at the edges of the words that
a record is cut into, for short lists and for lists too long for byte counts."""
import numpy as np
import pytest

import geneva_b200 as gv


@pytest.mark.gpu
@pytest.mark.parametrize("labels", [1, 4, 5, 8, 9, 12, 13, 27, 28, 29])
def test_segments_of_every_label(native, oracle, labels):
    rng = np.random.default_rng(labels)
    n = 1500
    lab = np.zeros(n + 1, dtype=np.uint32)
    lab[1:] = 1 + rng.integers(0, labels, n)
    lab[1:labels + 1] = 1 + np.arange(labels)
    # vertex 1 has 255 neighbours, vertex 2 256 and vertex 3 700; the others few
    pairs = {(1, v) for v in range(100, 355)} | {(2, v) for v in range(400, 656)} | {(3, v) for v in range(700, 1400)}
    for a, b in rng.integers(4, 90, (300, 2)):
        if a != b:
            pairs.add((min(a, b), max(a, b)))
    e = np.array(sorted(pairs), dtype=np.uint32)
    src, dst, el = e[:, 0].copy(), e[:, 1].copy(), np.ones(len(e), dtype=np.uint32)
    db, og = gv.Database.from_edges(lab, src, dst, el), oracle.from_edges(lab, src, dst, el)
    texts = [f"v 0 {a}\nv 1 {b}\ne 0 1 1\n" for a in range(1, labels + 1) for b in sorted({1, a, labels, 1 + a % labels})]
    plans = [gv.Plan.from_text(t) for t in texts]
    want = [len(oracle.match(og, t)[0]) for t in texts]
    assert sum(want) > 0
    got, _, _ = gv.batch_count(db, plans)
    assert [int(c) for c in got] == want
    assert [gv.match(db, p).num_rows for p in plans] == want
    oracle.free(og)
    db.close()
