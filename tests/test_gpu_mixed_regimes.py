"""Batches of several graphs in each regime of the planner's rule (chains per SM,
how the vertices are spread over the graphs): the plan is the regime's, and the
results stay those of a standalone call."""
import numpy as np
import pytest

from conftest import chains_for

pytestmark = pytest.mark.gpu

SIX = [("er", 700), ("er", 900), ("torus", 1200), ("er", 1200), ("tree", 1500), ("er", 500), ("torus", 14000)]
# graphs, chains of each, launch classes at least and at most, threads per chain of the largest class (None: any)
PLANS = {
    # up to two chains per SM: rows in HBM
    "few": ([("er", 700), ("torus", 14000)], 20, 1, 2, None),
    # up to 5.25: four warps for all
    "some": ([("er", 700), ("torus", 5000), ("tree", 9000)], 150, 1, 1, 128),
    # the same, one graph's chains most of the work: together
    "some_one": ([("er", 700), ("torus", 14000)], 300, 2, 4, None),
    "some_one_of_seven": (SIX, 80, 2, 4, None),
    # up to nine, and uneven graphs up to twelve: four warps for all
    "twelve_uneven": (SIX, 220, 1, 1, 128),
    # even ones: together
    "twelve_even": ([("er", 4200), ("torus", 4500), ("tree", 4900)], 540, 1, 4, None),
    # from sixteen on: rows in HBM, widths as they are
    "many": ([("er", 300), ("torus", 4200)], 1250, 1, 2, None),
}


@pytest.mark.parametrize("name", sorted(PLANS))
def test_regime(rfmf, ctx, name):
    graphs, C, least, most, threads = PLANS[name]
    dgs, gl, init, solver, t0s, sets = [], [], [], [], [], []
    for k, (kind, n) in enumerate(graphs):
        g = (rfmf.torus(n // 100, 100, signed=True, seed=k) if kind == "torus" else
             rfmf.random_tree(n, signed=True, seed=k) if kind == "tree" else
             rfmf.erdos_renyi_degree(n, 9, signed=True, seed=k))
        i, s = chains_for(g, [1000 * k + c % 7 for c in range(C)])
        s = [(x + 13 * c) % 2**64 for c, x in enumerate(s)]
        t = [(35.0, 70.0, 200.0, 400.0)[c % 4] for c in range(C)]
        dgs.append(rfmf.DeviceGraph(ctx, g))
        sets.append((g, i, t, s))
        gl += [dgs[-1]] * C
        init += list(i)
        solver += s
        t0s += t
    ph, it = [128, 16, 1], [6, 4, 5]
    b = rfmf.Batch(ctx, gl, t0s, solver, init, ph, it)
    info = b.info()
    if ctx.info()["sm_count"] == 152:
        assert least <= info["launch_classes"] <= most, info
        assert threads is None or info["threads_per_chain"] == threads, info
    b.run(9)
    b.run(6)
    r = b.read()
    b.close()
    for k, (g, i, t, s) in enumerate(sets):
        a = rfmf.anneal_gpu(ctx, dgs[k], g.max_weighted_degree(), i, t, ph, it, s)
        part = slice(k * C, (k + 1) * C)
        assert np.array_equal(r["cur_vals"][part], a.final_vals) and np.array_equal(r["best_vals"][part], a.best_vals)
        assert np.array_equal(np.stack(r["end_spins"][part]), a.end_spins)
        assert np.array_equal(np.stack(r["best_spins"][part]), a.best_spins)
        dgs[k].close()
