"""Rows read back to memory that the driver knows and memory that it doesn't,
on both sides of the size from which pieces go through pinned memory (8 MiB:
1,182 leaves give 8,375,652 bytes, 1,183 give 8,389,836) and of the 64 MiB after
which that memory is used again (3,345 leaves)."""
import ctypes

import numpy as np
import pytest
import torch

import geneva_b200 as gv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaves", [700, 1182, 1183, 3345])
def test_destinations(native, leaves):
    labels = np.array([0, 1] + [2] * leaves, np.uint32)
    leaf = np.arange(2, 2 + leaves, dtype=np.uint32)
    db = gv.Database.from_edges(labels, np.ones(leaves, np.uint32), leaf, np.ones(leaves, np.uint32))
    res = gv.match(db, gv.Plan.from_text("v 0 1\nv 1 2\nv 2 2\ne 0 1 1\ne 0 2 1\n"))
    n = leaves * (leaves - 1) // 2
    assert res.num_rows == n
    i, j = np.tril_indices(leaves, -1)
    want = np.sort(np.stack([leaf[j], leaf[i]], axis=1), axis=1)
    want = want[np.lexsort(want.T[::-1])]
    for pinned in (False, True):
        out = torch.full((n + 2, 3), 0x5a5a5a5a, dtype=torch.int32, pin_memory=pinned)
        rc = gv.library().gva_result_copy_rows(res._h, ctypes.c_void_p(out[1:].data_ptr()), 0, n)
        assert rc == 0
        rows = out.numpy().view(np.uint32)
        assert (rows[0] == 0x5a5a5a5a).all() and (rows[-1] == 0x5a5a5a5a).all()
        rows = rows[1:-1]
        assert (rows[:, 0] == 1).all()
        pairs = np.sort(rows[:, 1:], axis=1)
        assert np.array_equal(pairs[np.lexsort(pairs.T[::-1])], want)
    db.close()
