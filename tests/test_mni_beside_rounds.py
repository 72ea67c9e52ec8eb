"""An MNI run that may take half of the device leaves room for rounds on another
stream: they don't wait for its launches to end."""
import threading
import time

import numpy as np
import pytest
import torch

import geneva_b200 as gv
from geneva_b200 import workloads

pytestmark = pytest.mark.gpu


def test_rounds_run_beside_a_mining_run(native):
    db = workloads.graph_database(2000, 20, 60, 4.0, 4, None, 2, seed=8, name="beside")
    gdb = gv.Database.from_edges(db.vlabels, db.src, db.dst, db.elabels)
    gdb.set_graphs(db.first)
    plans = [gv.Plan.from_text(t) for t in workloads.sample_patterns(db, 16, 7, 10, seed=6)]
    g = workloads.rmat_graph(19, 16 << 19, 32, 1.0, seed=2, name="mined")
    mdb = gv.Database.from_edges(g.vlabels, g.src, g.dst, g.elabels)
    rounds, mining = torch.cuda.Stream(priority=-1), torch.cuda.Stream()

    def call():
        t0 = time.perf_counter()
        counts, _, _ = gv.batch_count(gdb, plans, stream=rounds.cuda_stream, support=True, host_rounds=True)
        return time.perf_counter() - t0, int(counts.sum())

    def mine():
        gv.mine(mdb, 5, 10000, support="mni", stream=mining.cuda_stream, sm_percent=50)

    mine()  # first launches and allocations
    want = call()[1]
    alone = [call()[0] for _ in range(200)]
    beside, over = [], threading.Event()

    def runs():
        try:
            for _ in range(2):
                mine()
        finally:
            over.set()

    miner = threading.Thread(target=runs)
    miner.start()
    while not over.is_set():
        t, n = call()
        beside.append(t)
        assert n == want
    miner.join()
    a, b = np.percentile(alone, 90) * 1e3, np.percentile(beside, 90) * 1e3
    # launches of the mining run last milliseconds; a call takes tenths of one
    assert b < 4 * a + 0.5
    gdb.close()
    mdb.close()
