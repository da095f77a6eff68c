"""Chains per CTA asked for with the chain width left to the planner: every
count up to 16 is planned, at a width that leaves room for it, whatever the
chain count and the graphs would have the planner choose."""
import numpy as np
import pytest

from conftest import chains_for

pytestmark = pytest.mark.gpu

# (graphs, chains of each): one graph at widths 8, 4, 2 and 1; phases that
# widen; several graphs in their regimes of two, four and twelve chains per SM
PLANS = {
    "wide": [("torus", 17000, 20)],
    "four": [("er", 2000, 600)],
    "two": [("er", 2000, 700)],
    "one": [("er", 900, 1900)],
    "rows": [("er", 600, 40)],
    "few": [("torus", 6000, 30), ("er", 700, 60)],
    "some": [("torus", 6000, 300), ("er", 700, 300)],
    "together": [("torus", 6000, 400), ("er", 700, 700)],
}


@pytest.mark.parametrize("name", sorted(PLANS))
def test_every_count_is_planned(rfmf, ctx, name):
    dgs, gl, init, solver, t0s = [], [], [], [], []
    for k, (kind, n, C) in enumerate(PLANS[name]):
        g = (rfmf.torus(n // 100, 100, signed=True, seed=k) if kind == "torus"
             else rfmf.erdos_renyi_degree(n, 20, signed=True, seed=k))
        i, s = chains_for(g, list(range(1000 * k, 1000 * k + C)))
        dgs.append(rfmf.DeviceGraph(ctx, g))
        gl += [dgs[-1]] * C
        init += list(i)
        solver += s
        t0s += [(35.0, 70.0, 200.0, 400.0)[c % 4] for c in range(C)]
    want = None
    for k in (0, 1, 2, 3, 4, 8, 9, 16):
        b = rfmf.Batch(ctx, gl, t0s, solver, init, [128, 8, 1], [3, 3, 3], rfmf.make_config(chains_per_cta=k))
        assert b.info()["threads_per_chain"] * max(k, 1) <= 512
        b.run(9)
        r = b.read()
        b.close()
        if want is None:
            want = r
        assert np.array_equal(r["cur_vals"], want["cur_vals"]) and np.array_equal(r["best_vals"], want["best_vals"])
        assert all(np.array_equal(x, y) for x, y in zip(r["end_spins"], want["end_spins"]))
    with pytest.raises(rfmf.RfmfError) as ei:
        rfmf.Batch(ctx, gl, t0s, solver, init, [128, 8, 1], [3, 3, 3], rfmf.make_config(chains_per_cta=17))
    assert ei.value.code == 1
    for dg in dgs:
        dg.close()
