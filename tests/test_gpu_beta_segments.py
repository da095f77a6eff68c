"""Betas of up to 32 sweeps held in the lanes of a warp: runs of one sweep, of a
few, of just around 32 and of hundreds, cut by windows and phases at every
offset, against the oracle bit for bit (integer work: tolerance zero)."""
import numpy as np
import pytest

from conftest import chains_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [32, 128])
@pytest.mark.parametrize("windows", [[10**6], [1, 31, 32, 33, 7, 64, 95, 700, 10**6]], ids=["one", "cut"])
def test_beta_runs_of_every_length(rfmf, ctx, oracle, threads, windows):
    g = rfmf.erdos_renyi_degree(150, 6, signed=True, seed=9)
    # runs at sweep s last about max(1, s t0 / 2^20) sweeps
    t0s = [35.0, 3000.0, 2.0e4, 1.0e6, 3.0e7]
    init, solver = chains_for(g, [11, 12, 13, 14, 15])
    ph, it = [16, 3, 0, 1], [45, 1500, 10, 1000]
    dg = rfmf.DeviceGraph(ctx, g)
    b = rfmf.Batch(ctx, [dg] * 5, t0s, solver, init, ph, it, rfmf.make_config(threads_per_chain=threads))
    left = 2545
    for w in windows:
        b.run(min(w, left))
        left -= min(w, left)
    r = b.read()
    b.close()
    dg.close()
    o = oracle.anneal(g, init, t0s, solver, ph, it)
    assert left == 0
    assert np.array_equal(r["cur_vals"], o["cur_vals"])
    assert np.array_equal(r["best_vals"], o["best_vals"])
    assert np.array_equal(np.stack(r["end_spins"]), o["end_spins"])
    assert np.array_equal(np.stack(r["best_spins"]), o["best_spins"])
