"""Several graphs side by side, as requests of one window and as one batch: each
runs at a width chosen with the others' and, from 4096 vertices on, walks its
rows in HBM.  The results must stay those of a standalone call."""
import numpy as np
import pytest

from conftest import chains_for

pytestmark = pytest.mark.gpu

MIXES = {
    # the largest graph wide, the small ones narrow; both sides of 4096 vertices
    "sizes": [("torus", 4095, 40, 1), ("torus", 4100, 30, 1), ("torus", 14000, 12, 1), ("er", 700, 200, 1),
              ("er", 65, 3, 1)],
    # a copy that leaves little room beside a class mate's larger chains
    "crowded": [("dense", 1200, 2, 1), ("torus", 4000, 2, 1), ("er", 900, 1, 1)],
    # int32 gains and 32-bit entries beside int8
    "weights": [("er", 900, 24, 300), ("torus", 5000, 24, 1), ("torus", 5000, 16, 300)],
    # one schedule off the kernel's main path (P = 300) beside two on it
    "table": [("er", 500, 30, 1), ("torus", 14000, 12, 1), ("torus", 4100, 20, 1)],
    # more than ten chains per SM: the requests' own widths, several classes
    "many": [("er", 300, 900, 1), ("torus", 4200, 300, 1), ("er", 600, 800, 40)],
}


def _graph(rfmf, kind, n, wmax, seed):
    if kind == "torus":
        rows = next(k for k in range(int(n ** 0.5), 0, -1) if n % k == 0)
        g = rfmf.torus(rows, n // rows, signed=True, seed=seed)
    else:
        g = rfmf.erdos_renyi_degree(n, 8 if kind == "er" else 76, signed=True, seed=seed)
    if wmax > 1:
        rng = np.random.default_rng(seed)
        m = {}
        src = np.repeat(np.arange(g.n), np.diff(g.offsets.astype(np.int64)))
        w = np.empty_like(g.weight)
        for i, (a, b) in enumerate(zip(src, g.col)):
            key = (min(a, b), max(a, b))
            if key not in m:
                m[key] = int(rng.integers(1, wmax + 1)) * (1 if rng.random() < 0.5 else -1)
            w[i] = m[key]
        g.weight = w
    return g


@pytest.mark.parametrize("name", sorted(MIXES))
def test_mixed_requests_match_standalone(rfmf, ctx, name):
    srv = rfmf.Server(ctx, window_sweeps=37)
    reqs = []
    for k, (kind, n, C, wmax) in enumerate(MIXES[name]):
        g = _graph(rfmf, kind, n, wmax, 11 + k)
        init, solver = chains_for(g, list(range(1000 * k, 1000 * k + C)))
        t0s = [(35.0, 70.0, 200.0, 400.0)[c % 4] * (1 if wmax == 1 else 100) for c in range(C)]
        reqs.append((g, rfmf.DeviceGraph(ctx, g), init, solver, t0s, [300 if name == "table" and k == 0 else 128, 16, 1],
                     [40 + 30 * k, 25, 20]))
    ids = [srv.submit(dg, init, t0s, ph, it, solver) for _, dg, init, solver, t0s, ph, it in reqs]
    for rid, (g, dg, init, solver, t0s, ph, it) in zip(ids, reqs):
        st = srv.wait(rid, timeout=300)
        assert st["state"] == "done"
        a = srv.result(rid)
        b = rfmf.anneal_gpu(ctx, dg, g.max_weighted_degree(), init, t0s, ph, it, solver)
        assert np.array_equal(a.end_spins, b.end_spins)
        assert np.array_equal(a.best_spins, b.best_spins)
        assert np.array_equal(a.best_vals, b.best_vals)
        assert np.array_equal(a.final_vals, b.final_vals)


@pytest.mark.parametrize("wmax", [1, 60])
def test_mixed_batch_matches_standalone(rfmf, ctx, wmax):
    # between 5.25 and 12 chains per SM: widths chosen together
    mix = [("torus", 4100, 300, wmax), ("torus", 14000, 40, 1), ("er", 700, 520, wmax)]
    sets, dgs, init, solver, t0s = [], [], [], [], []
    for k, (kind, n, C, w) in enumerate(mix):
        g = _graph(rfmf, kind, n, w, 31 + k)
        dg = rfmf.DeviceGraph(ctx, g)
        i, s = chains_for(g, list(range(1000 * k, 1000 * k + C)))
        t = [(35.0, 70.0, 200.0, 400.0)[c % 4] * (1 if w == 1 else 50) for c in range(C)]
        sets.append((g, dg, i, s, t))
        dgs += [dg] * C
        init += list(i)
        solver += list(s)
        t0s += t
    ph, it = [128, 16, 1], [40, 25, 20]
    b = rfmf.Batch(ctx, dgs, t0s, solver, init, ph, it)
    for sweeps in (13, 40, 32):   # windows that cut phases
        b.run(sweeps)
    r = b.read()
    b.close()
    at = 0
    for g, dg, i, s, t in sets:
        a = rfmf.anneal_gpu(ctx, dg, g.max_weighted_degree(), i, t, ph, it, s)
        C = len(t)
        assert np.array_equal(np.stack(r["end_spins"][at:at + C]), a.end_spins)
        assert np.array_equal(np.stack(r["best_spins"][at:at + C]), a.best_spins)
        assert np.array_equal(r["best_vals"][at:at + C], a.best_vals)
        assert np.array_equal(r["cur_vals"][at:at + C], a.final_vals)
        at += C
