"""Two requests whose chains fill nearly all of the SMs' shared memory: beside
each other at widths chosen together they would come in rounds, so they run at
their own; results equal standalone calls."""
import numpy as np
import pytest

from conftest import chains_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [640, 750])
def test_full_shared_memory(rfmf, ctx, C):
    reqs = []
    for k, g in enumerate((rfmf.random_tree(10000, signed=True, seed=1), rfmf.torus(70, 100, signed=True, seed=2))):
        i, s = chains_for(g, [100 * k + c % 5 for c in range(C)])
        s = [(x + 17 * c) % 2**64 for c, x in enumerate(s)]
        reqs.append((g, rfmf.DeviceGraph(ctx, g), i, [(50.0, 200.0)[c % 2] for c in range(C)], [128, 1], [6, 5], s))
    srv = rfmf.Server(ctx, window_sweeps=3)
    ids = [srv.submit(*r[1:]) for r in reqs]
    for rid in ids:
        assert srv.wait(rid, timeout=300)["state"] == "done"
    for rid, (g, dg, i, t, ph, it, s) in zip(ids, reqs):
        got, want = srv.result(rid), rfmf.anneal_gpu(ctx, dg, g.max_weighted_degree(), i, t, ph, it, s)
        assert np.array_equal(got.end_spins, want.end_spins) and np.array_equal(got.best_vals, want.best_vals)
        assert np.array_equal(got.best_spins, want.best_spins) and np.array_equal(got.final_vals, want.final_vals)
        dg.close()
    srv.close()
