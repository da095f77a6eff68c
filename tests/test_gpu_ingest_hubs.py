"""Hub rows of the device ingest (above 2048 entries: tiles sorted and merged)
at the edges of their tiles and merge passes, against the host CSR bit for bit;
and the time of a long one, which must not grow as its square."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _stars(degrees, order, seed):
    """One star per degree over shared leaves, one line in five repeated with
    another weight and the other orientation."""
    rng = np.random.default_rng(seed)
    u = np.concatenate([np.full(d, 2 * c) for c, d in enumerate(degrees)])
    v = np.concatenate([1000 + rng.permutation(max(degrees) + 9)[:d] for d in degrees])
    if order == "ascending":
        k = np.lexsort((v, u))
    elif order == "descending":
        k = np.lexsort((-v, -u))
    else:
        k = rng.permutation(len(u))
    u, v = u[k], v[k]
    w = rng.integers(1, 300, len(u))
    again = np.arange(0, len(u), 5)
    return np.concatenate([u, v[again]]), np.concatenate([v, u[again]]), np.concatenate([w, -w[again]])


@pytest.mark.parametrize("order", ["ascending", "descending", "random"])
@pytest.mark.parametrize("degrees", [(1707,), (2049, 2048, 2047), (3413, 4096, 4097, 10), (6144, 6145, 3000, 8191, 8193),
                                     (100001, 5000, 70000), (2100,) * 400], ids=lambda d: f"{len(d)}x{d[0]}")
def test_hub_rows(rfmf, ctx, degrees, order):
    u, v, w = _stars(degrees, order, sum(degrees))
    ref = rfmf.csr_from_edges(u, v, w)
    g = rfmf.DeviceGraph.from_edges(ctx, u, v, w)
    off, col, wt = g.csr()
    assert np.array_equal(off, ref.offsets) and np.array_equal(col, ref.col) and np.array_equal(wt, ref.weight)
    assert np.array_equal(g.orig_ids(), ref.orig_ids)
    assert g.info() == dict(n=ref.n, m=ref.m, max_weighted_degree=ref.max_weighted_degree())
    g.close()


def test_long_hub_is_quick(rfmf, ctx):
    # 300,000 keys ranked against each other are 9e10 comparisons, over a second
    # on one SM; sorted, a few ms beside the copies
    u, v, w = _stars((300000,), "random", 1)
    rfmf.DeviceGraph.from_edges(ctx, u[:1000], v[:1000], w[:1000]).close()
    t0 = time.perf_counter()
    rfmf.DeviceGraph.from_edges(ctx, u, v, w).close()
    assert time.perf_counter() - t0 < 0.25
