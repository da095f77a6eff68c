"""Requests on one graph that read it in different CSR formats, in flight
together: a request of many chains leaves no room for a shared-memory copy and
walks HBM, one of a single chain stages it.  Each must equal its standalone
call, whichever was admitted first."""
import time

import numpy as np
import pytest

from conftest import chains_for

pytestmark = pytest.mark.gpu


def _graph(rfmf, kind):
    # By the planner's formulas on 152 SMs with 227 KB of shared memory: 256
    # chains need 247,680 B (tree) or 240,080 B (torus), one chain 211,776 or
    # 204,176 B.
    return rfmf.random_tree(14000, signed=True, seed=3) if kind == "tree" else rfmf.torus(100, 140, signed=True, seed=3)


@pytest.mark.parametrize("kind", ["tree", "torus"])
@pytest.mark.parametrize("first", ["many", "one"])
def test_two_formats_of_one_graph(rfmf, ctx, kind, first):
    g = _graph(rfmf, kind)
    dg = rfmf.DeviceGraph(ctx, g)
    reqs = []
    for C, seed, it in ((256, 0, [300, 200, 100]), (1, 900, [40, 30, 20])):
        init, solver = chains_for(g, list(range(seed, seed + C)))
        reqs.append((init, [(35.0, 70.0, 200.0, 400.0)[c % 4] for c in range(C)], [128, 16, 1], it, solver))
    if first == "one":
        reqs = [(reqs[1][0], reqs[1][1], [128, 16, 1], [3000, 2000, 1000], reqs[1][4]),
                (reqs[0][0], reqs[0][1], [128, 16, 1], [40, 30, 20], reqs[0][4])]
    alone = [rfmf.anneal_gpu(ctx, dg, g.max_weighted_degree(), i, t, p, it, s) for i, t, p, it, s in reqs]
    srv = rfmf.Server(ctx, window_sweeps=5)
    ids = [srv.submit(dg, *reqs[0])]
    while srv.poll(ids[0])["state"] == "queued":
        time.sleep(1e-4)
    ids.append(srv.submit(dg, *reqs[1]))
    st = [srv.wait(i, timeout=300) for i in ids]
    assert [s["state"] for s in st] == ["done", "done"]
    assert st[1]["start_s"] < st[0]["finish_s"]   # they did run side by side
    for rid, want in zip(ids, alone):
        got = srv.result(rid)
        assert np.array_equal(got.end_spins, want.end_spins)
        assert np.array_equal(got.best_spins, want.best_spins)
        assert np.array_equal(got.best_vals, want.best_vals)
        assert np.array_equal(got.final_vals, want.final_vals)
    srv.close()
    dg.close()
