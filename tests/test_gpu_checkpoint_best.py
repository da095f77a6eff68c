"""A checkpoint whose best cut lies below its current one: best moves after a
sweep only, to that sweep's cut, so resuming and running nothing changes
nothing, and the state resumed from is never taken for a sweep's result."""
import numpy as np
import pytest

from conftest import chains_for

pytestmark = pytest.mark.gpu

PHASES, ITERS = [16, 4, 1], [40, 300, 300]


@pytest.mark.parametrize("threads", [32, 128])
@pytest.mark.parametrize("wmax", [1, 60], ids=["int8_gains", "int32_gains"])
@pytest.mark.parametrize("piece", [1, 100])
@pytest.mark.parametrize("replay", [False, True], ids=["run", "run_graph"])
def test_best_below_current(rfmf, ctx, threads, wmax, piece, replay):
    g = rfmf.erdos_renyi_degree(300, 8, signed=True, seed=5)
    g.weight = g.weight * wmax
    seeds = list(range(12))
    init, solver = chains_for(g, seeds)
    # t0 from cold to hot: with cold ones the first sweeps' cuts stay below the
    # one resumed from, with hot ones they pass it
    t0s = [(20.0, 100.0, 400.0)[c % 3] * wmax for c in seeds]
    cfg = rfmf.make_config(threads_per_chain=threads)
    dg = rfmf.DeviceGraph(ctx, g)
    gl = [dg] * len(seeds)
    b = rfmf.Batch(ctx, gl, t0s, solver, init, PHASES, ITERS, cfg)
    b.run(200)
    state = b.read()
    b.close()
    low = dict(state, best_spins=list(init),
               best_vals=np.array([rfmf.cut_value(g, s) for s in init], np.int64))
    assert (low["best_vals"] < low["cur_vals"]).all()

    b = rfmf.Batch.restore(ctx, gl, t0s, solver, PHASES, ITERS, low, cfg)
    b.run(0)
    b.run_graph(0)
    r = b.read()
    assert np.array_equal(r["cur_vals"], low["cur_vals"]) and np.array_equal(r["best_vals"], low["best_vals"])
    assert all(np.array_equal(x, y) for x, y in zip(r["best_spins"], low["best_spins"]))
    assert not b.improved_sweeps().any()

    # sweep by sweep, from the current cuts alone
    best, spins = low["best_vals"].copy(), list(low["best_spins"])
    improved = np.zeros(len(seeds), np.uint64)
    one = rfmf.Batch.restore(ctx, gl, t0s, solver, PHASES, ITERS, low, cfg)
    end = 200 + 2 * piece
    for _ in range(200, end):
        one.run(1)
        s = one.read()
        for c in range(len(seeds)):
            if s["cur_vals"][c] > best[c]:
                best[c], spins[c] = s["cur_vals"][c], s["end_spins"][c].copy()
                improved[c] += 1
    one.close()
    if replay:
        b.run_graph(piece, launches=1, replays=2)
    else:
        b.run(piece)
        b.run(piece)
    r = b.read()
    assert (r["sweeps_done"] == end).all()
    assert np.array_equal(r["best_vals"], best)
    assert all(np.array_equal(x, y) for x, y in zip(r["best_spins"], spins))
    assert np.array_equal(b.improved_sweeps(), improved)
    b.close()
    dg.close()
