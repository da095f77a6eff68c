"""rfmf_graph_csr reads a graph back while anneals are queued on its context: it
neither waits for them nor needs the SMs they fill."""
import time

import numpy as np
import pytest

from conftest import chains_for

pytestmark = pytest.mark.gpu


def test_csr_does_not_wait_for_queued_windows(rfmf, ctx):
    g = rfmf.erdos_renyi_degree(2000, 19, signed=True, seed=1)
    dg = rfmf.DeviceGraph(ctx, g)
    init, solver = chains_for(g, list(range(64)))
    init, solver = np.tile(init, (32, 1)), solver * 32   # 2048 chains: every SM is full
    b = rfmf.Batch(ctx, [dg] * 2048, [100.0] * 2048, solver, list(init), [16, 1], [100000, 100000])
    dg.csr()
    b.run(20)
    b.read()
    t0 = time.perf_counter()
    for _ in range(4):
        b.run(20000)
    off, col, w = dg.csr()
    t_csr = time.perf_counter() - t0
    b.read()
    t_all = time.perf_counter() - t0
    b.close()
    dg.close()
    assert np.array_equal(off, g.offsets) and np.array_equal(col, g.col) and np.array_equal(w, g.weight)
    assert t_csr < t_all / 4, (t_csr, t_all)


@pytest.mark.parametrize("m", [1, 65535, 65536, 65537, 150000])
def test_parts(rfmf, ctx, m):
    # two entries an edge: lengths around the parts it is copied in
    n = m + 1
    u, v = np.arange(m), np.arange(1, n)
    w = np.random.default_rng(m).integers(1, 1000, m)
    dg = rfmf.DeviceGraph.from_edges(ctx, u, v, w)
    off, col, wt = dg.csr()
    want = rfmf.csr_from_edges(u, v, w)
    assert np.array_equal(off, want.offsets) and np.array_equal(col, want.col) and np.array_equal(wt, want.weight)
    dg.close()
