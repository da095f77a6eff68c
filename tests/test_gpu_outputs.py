"""Cuts and partition strings recomputed on the device, against the spins and
the host's cut of them: groups of 32 chains and remainders, weights from +-1
to 2^27, graphs that fit the
vertex table of a CTA and one that does not, row strides off 16 bytes."""
import ctypes as ct

import numpy as np
import pytest

from conftest import chains_for

pytestmark = pytest.mark.gpu


def _weighted(rfmf, wmax):
    rng = np.random.default_rng(wmax)
    u, v = np.arange(200), (np.arange(200) + 1) % 200
    w = rng.integers(1, wmax + 1, 200) * rng.choice([-1, 1], 200)
    return rfmf.csr_from_edges(u, v, w)


@pytest.mark.parametrize("extra", [0, 1, 13])
def test_cuts_and_partitions(rfmf, ctx, extra):
    graphs = [rfmf.erdos_renyi(33, 0.3, signed=True, seed=1), rfmf.erdos_renyi_sparse(1000, 6, signed=True, seed=2),
              rfmf.random_tree(60001, signed=True, seed=3), _weighted(rfmf, 3), _weighted(rfmf, 2**27)]
    counts = [33, 64, 3, 40, 5]
    dgs = [rfmf.DeviceGraph(ctx, g) for g in graphs]
    which, gl, ini, sol = [], [], [], []
    for k, (g, c) in enumerate(zip(graphs, counts)):
        init, solver = chains_for(g, list(range(100 * k, 100 * k + c)))
        for i in range(c):
            which.append(k)
            ini.append(init[i])
            sol.append(solver[i])
    order = np.random.default_rng(4).permutation(len(which))   # chains of the graphs interleaved
    which, ini, sol = [which[i] for i in order], [ini[i] for i in order], [sol[i] for i in order]
    gl = [dgs[k] for k in which]
    b = rfmf.Batch(ctx, gl, [60.0 * (2.0**27 if k == 4 else 1.0) for k in which], sol, ini, [4, 1], [30, 30])
    b.run(60)
    r = b.read()
    stride = max(g.n for g in graphs) + extra
    text = np.full((len(gl), stride), 255, np.uint8)
    for best in (False, True):
        spins = r["best_spins" if best else "end_spins"]
        want = [rfmf.cut_value(graphs[k], s) for k, s in zip(which, spins)]
        assert b.cuts(best=best).tolist() == want
        assert rfmf.lib().rfmf_batch_partitions(b.h, int(best), ct.c_void_p(text.ctypes.data), stride) == 0
        for row, k, s in zip(text, which, spins):
            n = graphs[k].n
            assert np.array_equal(row[:n], np.where(s > 0, ord("1"), ord("0")))
            assert not row[n:].any()
    b.close()
    for dg in dgs:
        dg.close()
