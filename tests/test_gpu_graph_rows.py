"""Compact rows made from a host CSR (rfmf_graph_create): rows of zero to nine
entries in every order, isolated vertices at the front, in between and at the
end, long stretches without padding.  An anneal on each compact form must equal
the one on the 8-byte pairs, and the CSR reads back as it was."""
import numpy as np
import pytest

from conftest import chains_for

pytestmark = pytest.mark.gpu


def _csr(rfmf, n, pairs, rng, wmax):
    """A graph over exactly n vertices (isolated ones kept)."""
    rows = [[] for _ in range(n)]
    for a, b in pairs:
        w = int(rng.integers(1, wmax + 1)) * (1 if rng.random() < 0.5 else -1)
        rows[a].append((b, w))
        rows[b].append((a, w))
    off, col, wt = [0], [], []
    for r in rows:
        for c, w in sorted(r):
            col.append(c)
            wt.append(w)
        off.append(len(col))
    g = rfmf.torus(3, 3, seed=1)
    g.n, g.offsets, g.col, g.weight = n, np.array(off, np.uint32), np.array(col, np.int32), np.array(wt, np.int32)
    g.orig_ids = np.arange(n)
    return g


def _pairs(kind, rng):
    if kind == "sparse":        # degrees 0 to about 9, isolated ends
        n = 300
        p = {tuple(sorted(rng.integers(5, n - 7, 2).tolist())) for _ in range(600)}
    elif kind == "regular":     # a torus: rows of four, no padding, then a path
        n = 400
        p = {tuple(sorted((20 * i + j, 20 * ((i + 1) % 10) + j))) for i in range(10) for j in range(20)}
        p |= {tuple(sorted((20 * i + j, 20 * i + (j + 1) % 20))) for i in range(10) for j in range(20)}
        p |= {(k, k + 1) for k in range(210, 399)}
    elif kind == "star":        # one long row among rows of one, the last vertex its centre
        n = 103
        p = {(k, 102) for k in range(1, 99)}
    elif kind == "pair":        # fewer entries than a vector
        n, p = 6, {(2, 4)}
    else:                       # the last rows end within a vector of the arrays' end
        n = 50
        p = {(k, k + 1) for k in range(0, 49)} | {(0, 47), (1, 48), (2, 49)}
    return n, sorted(x for x in p if x[0] != x[1])


@pytest.mark.parametrize("wmax", [1, 30])
@pytest.mark.parametrize("kind", ["sparse", "regular", "star", "pair", "path"])
def test_rows(rfmf, ctx, oracle, kind, wmax):
    rng = np.random.default_rng(len(kind))
    n, pairs = _pairs(kind, rng)
    g = _csr(rfmf, n, pairs, rng, wmax)
    dg = rfmf.DeviceGraph(ctx, g)
    off, col, w = dg.csr()
    assert np.array_equal(off, g.offsets) and np.array_equal(col, g.col) and np.array_equal(w, g.weight)
    B = rfmf.max_weighted_degree(g)
    init, solver = chains_for(g, [1, 2, 3])
    t0s, ph, it = [30.0 * wmax, 100.0 * wmax, 300.0 * wmax], [8, 3, 1], [20, 20, 20]
    o = oracle.anneal(g, init, t0s, solver, ph, it)
    for fmt in ([1] if wmax == 1 else []) + [0, 2, 3, 4]:
        for gain in (0, 4):
            for threads in (32, 64):
                r = rfmf.anneal_gpu(ctx, dg, B, init, t0s, ph, it, solver,
                                    rfmf.make_config(csr_format=fmt, gain_width=gain, threads_per_chain=threads))
                assert np.array_equal(r.end_spins, o["end_spins"]), (fmt, gain, threads)
                assert np.array_equal(r.best_vals, o["best_vals"]) and np.array_equal(r.final_vals, o["cur_vals"])
    dg.close()


@pytest.mark.parametrize("n", [2, 32768, 32769, 32770, 100001])
def test_read_back_in_parts(rfmf, ctx, n):
    # a path: 2 (n - 1) entries, around the parts they are split in
    k = np.arange(n - 1)
    g = rfmf.csr_from_edges(k, k + 1, np.random.default_rng(n).integers(1, 1000, n - 1))
    dg = rfmf.DeviceGraph(ctx, g)
    off, col, w = dg.csr()
    assert np.array_equal(off, g.offsets) and np.array_equal(col, g.col) and np.array_equal(w, g.weight)
    dg.close()
