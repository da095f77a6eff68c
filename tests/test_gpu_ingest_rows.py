"""Device ingest at the edges of its row sort (a warp's 32 keys, the hub rows
that take a block, row padding) against the host CSR, and an anneal on the
built graph against the oracle (its compact rows), all bit for bit."""
import numpy as np
import pytest

from conftest import chains_for

pytestmark = pytest.mark.gpu


def _stars(degrees, wmax, seed):
    """One star per degree over shared leaves, every seventh edge repeated with
    another weight and the other orientation, zero-weight lines in between."""
    rng = np.random.default_rng(seed)
    u, v = [], []
    for c, d in enumerate(degrees):
        leaves = 1000 + rng.permutation(max(degrees) + 50)[:d]
        u.append(np.full(d, 3 * c))
        v.append(leaves)
    u, v = np.concatenate(u), np.concatenate(v)
    order = rng.permutation(len(u))
    u, v = u[order], v[order]
    w = rng.integers(1, wmax + 1, len(u)) * rng.choice([-1, 1], len(u))
    again = np.arange(0, len(u), 7)
    zero = np.arange(0, len(u), 11)
    return (np.concatenate([u, v[again], u[zero] + 1]), np.concatenate([v, u[again], v[zero]]),
            np.concatenate([w, -w[again], np.zeros(len(zero), np.int64)]).astype(np.int64))


@pytest.mark.parametrize("wmax", [1, 7, 40000])
@pytest.mark.parametrize("degrees", [(1, 2, 3, 4, 5), (31, 32, 33), (63, 64, 65, 127, 129), (2047, 2048, 2049),
                                     (9000, 2500, 3)], ids=str)
def test_rows_of_every_length(rfmf, ctx, oracle, degrees, wmax):
    u, v, w = _stars(degrees, wmax, sum(degrees))
    keep = w != 0
    ref = rfmf.csr_from_edges(u[keep], v[keep], w[keep])
    g = rfmf.DeviceGraph.from_edges(ctx, u, v, w)
    off, col, wt = g.csr()
    assert np.array_equal(off, ref.offsets) and np.array_equal(col, ref.col) and np.array_equal(wt, ref.weight)
    assert np.array_equal(g.orig_ids(), ref.orig_ids)
    assert g.info() == dict(n=ref.n, m=ref.m, max_weighted_degree=ref.max_weighted_degree())
    init, solver = chains_for(ref, [1, 2])
    t0s, phases, iters = [50.0 * wmax * len(degrees), 400.0 * wmax], [64, 5, 1], [6, 6, 6]
    r = rfmf.anneal_gpu(ctx, g, ref.max_weighted_degree(), init, t0s, phases, iters, solver)
    o = oracle.anneal(ref, init, t0s, solver, phases, iters)
    g.close()
    assert np.array_equal(r.end_spins, o["end_spins"]) and np.array_equal(r.best_vals, o["best_vals"])


def test_bad_lines_are_named_in_order(rfmf, ctx):
    """The first bad line decides the error, wherever the others are."""
    u = np.arange(0, 3000)
    v = u + 1
    w = np.ones(3000, np.int64)
    for neg, big, what in ((700, 900, "negative vertex id at edge 700"), (900, 700, "weight at edge 700"),
                           (700, 700, "negative vertex id at edge 700")):
        uu, ww = u.copy(), w.copy()
        uu[neg] = -5
        ww[big] = 2**31
        with pytest.raises(rfmf.RfmfError, match=what):
            rfmf.DeviceGraph.from_edges(ctx, uu, v, ww)
    loop = v.copy()
    loop[1500] = u[1500]
    with pytest.raises(rfmf.RfmfError, match="self loop"):
        rfmf.DeviceGraph.from_edges(ctx, u, loop, w)
    w[1500] = 0
    assert rfmf.DeviceGraph.from_edges(ctx, u, loop, w).info()["m"] == 2999
