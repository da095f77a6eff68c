"""Requests that fit a CTA each by itself, but not the largest need of one
beside the largest of another, in one window: they run as classes of their own,
and no request fails because of what shares its window."""
import numpy as np
import pytest

from conftest import chains_for

pytestmark = pytest.mark.gpu


def _serve(rfmf, ctx, reqs, window, **launch):
    srv = rfmf.Server(ctx, window_sweeps=window, cfg=rfmf.make_config(**launch))
    made = []
    for k, (g, C, ph, it) in enumerate(reqs):
        init, solver = chains_for(g, list(range(1000 * k, 1000 * k + C)))
        made.append((g, rfmf.DeviceGraph(ctx, g), init, [(300.0, 900.0)[c % 2] for c in range(C)], ph, it, solver))
    ids = [srv.submit(*m[1:]) for m in made]
    st = [srv.wait(i, timeout=300) for i in ids]
    assert [s["state"] for s in st] == ["done"] * len(st), [s["error"] for s in st]
    assert st[1]["start_s"] < st[0]["finish_s"]
    for rid, (g, dg, init, t0s, ph, it, solver) in zip(ids, made):
        got = srv.result(rid)
        want = rfmf.anneal_gpu(ctx, dg, g.max_weighted_degree(), init, t0s, ph, it, solver)
        assert np.array_equal(got.end_spins, want.end_spins)
        assert np.array_equal(got.best_spins, want.best_spins)
        assert np.array_equal(got.best_vals, want.best_vals)
        assert np.array_equal(got.final_vals, want.final_vals)
        dg.close()
    srv.close()


def test_many_vertices_beside_many_groups(rfmf, ctx):
    # 65,000 vertices with a few groups, 5,500 vertices with a group each: both
    # off the kernel's main path, four warps, 32-bit entries in HBM
    big, small = rfmf.random_tree(65000, seed=1), rfmf.random_tree(5500, seed=2)
    big.weight, small.weight = big.weight * 2, small.weight * 2
    _serve(rfmf, ctx, [(big, 305, [300, 1], [150, 50]), (small, 2, [5500, 1], [20, 10])], 4)


@pytest.mark.parametrize("fmt", [1, 2])
def test_large_copy_beside_large_chain(rfmf, ctx, fmt):
    # shared-memory copies asked for, of 215 to 225 KB: 8 KB of chain fit beside
    # one in a CTA's 227 KB, the other request's 18 KB do not
    dense = rfmf.erdos_renyi_degree(1700 if fmt == 1 else 900, 61 if fmt == 1 else 58, signed=True, seed=3)
    wide = rfmf.torus(60, 100, signed=True, seed=4)
    _serve(rfmf, ctx, [(dense, 1, [128, 1], [3000, 1000]), (wide, 1, [128, 1], [40, 20])], 50, csr_format=fmt)
