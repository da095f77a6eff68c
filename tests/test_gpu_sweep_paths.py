"""Every route of a sweep through the kernel against the oracle, bit for bit
(integer work: tolerance zero): group counts that reduce per warp, per thread
and per vertex, chain widths, gain widths, and vertex counts at the edges of a
warp's block loop (32 W blocks of 8 vertices an iteration, three iterations in
flight), and past the 16 iterations a one-warp chain's keys number in 4 bits."""
import numpy as np
import pytest

from conftest import chains_for

pytestmark = pytest.mark.gpu

PHASES = {
    "halving": [256, 128, 64, 32, 16, 8, 4, 2, 1],
    "odd": [200, 129, 100, 83, 60, 33, 31, 17, 12, 7, 5, 3],
}


def _graph(rfmf, n, wmax):
    """A cycle through all n vertices (so none is dropped) plus random chords."""
    rng = np.random.default_rng(n + wmax)
    m = 2 * n
    u = np.concatenate([np.arange(n), rng.integers(0, n, m)])
    v = np.concatenate([(np.arange(n) + 1) % n, rng.integers(0, n, m)])
    keep = u != v
    u, v = u[keep], v[keep]
    w = rng.integers(1, wmax + 1, len(u)) * rng.choice([-1, 1], len(u))
    return rfmf.csr_from_edges(u, v, w)


@pytest.mark.parametrize("wmax", [1, 4, 400], ids=["unit", "int8_gains", "int32_gains"])
@pytest.mark.parametrize("phases", sorted(PHASES))
@pytest.mark.parametrize("threads", [32, 64, 128, 256])
def test_sweep_routes(rfmf, ctx, oracle, threads, phases, wmax):
    sizes = [5, 255, 257, 8 * threads - 1, 24 * threads + 9, 32 * threads + 8]
    if threads == 32:
        sizes.append(4231)
    for n in sizes:
        g = _graph(rfmf, n, wmax)
        seeds, t0s = [3, 4, 5], [35.0 * wmax, 120.0 * wmax, 400.0 * wmax]
        init, solver = chains_for(g, seeds)
        ph = PHASES[phases]
        iters = [7] * len(ph)
        with_cfg = rfmf.make_config(threads_per_chain=threads)
        dg = rfmf.DeviceGraph(ctx, g)
        r = rfmf.anneal_gpu(ctx, dg, g.max_weighted_degree(), init, t0s, ph, iters, solver, with_cfg)
        o = oracle.anneal(g, init, t0s, solver, ph, iters)
        dg.close()
        where = f"n={n} threads={threads} {phases} wmax={wmax}"
        assert np.array_equal(r.final_vals, o["cur_vals"]), where
        assert np.array_equal(r.best_vals, o["best_vals"]), where
        assert np.array_equal(r.end_spins, o["end_spins"]), where
        assert np.array_equal(r.best_spins, o["best_spins"]), where
