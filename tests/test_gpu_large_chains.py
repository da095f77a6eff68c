"""Chains at the limit of a CTA's shared memory, through every entry point,
against the oracle bit for bit: without room for the argmax scratch (int32
scores through the group slots), at a narrower width than the planner's first
(with key room at that width and without), and copies asked for that fit a CTA
only with their rows packed (walked in HBM).  The sizes are the planner's own
limits for int8 gains and 227 KB of shared memory a CTA."""
import importlib

import numpy as np
import pytest

from conftest import chains_for

pytestmark = pytest.mark.gpu

# vertices, phases, t0
CASES = {
    "scratch": (99000, [128, 16, 1], 200.0),          # eight warps with scratch
    "slots": (102000, [128, 16, 1], 200.0),           # eight warps without
    "slots_any": (102000, [100, 128, 3], 200.0),
    "narrower": (103050, [16, 4, 1], 200.0),          # four warps only
    "narrower_no_keys": (103050, [16, 4, 1], 30.0),   # their keys at fewer warps lack room
    "one_warp_keys": (103160, [1, 1, 1], 30.0),
}


def _same(r, o):
    assert np.array_equal(r.final_vals, o["cur_vals"]) and np.array_equal(r.best_vals, o["best_vals"])
    assert np.array_equal(r.end_spins, o["end_spins"]) and np.array_equal(r.best_spins, o["best_spins"])


@pytest.mark.parametrize("name", sorted(CASES))
def test_every_entry_point(rfmf, ctx, oracle, name):
    n, ph, t0 = CASES[name]
    g = rfmf.random_tree(n, signed=True, seed=5)
    init, solver = chains_for(g, [1, 2])
    t0s, it = [t0, 2 * t0], [6, 5, 4]
    o = oracle.anneal(g, init, t0s, solver, ph, it)
    dg = rfmf.DeviceGraph(ctx, g)
    B = g.max_weighted_degree()
    _same(rfmf.anneal_gpu(ctx, dg, B, init, t0s, ph, it, solver), o)
    _same(rfmf.anneal_gpu(ctx, dg, B, init, t0s, ph, it, solver, rfmf.make_config(threads_per_chain=32)), o)
    srv = rfmf.Server(ctx, window_sweeps=4)
    rid = srv.submit(dg, init, t0s, ph, it, solver)
    assert srv.wait(rid, timeout=300)["state"] == "done"
    _same(srv.result(rid), o)
    srv.close()
    dg.close()
    rc, out = importlib.import_module("test_zz_no_alloc")._Caller(rfmf, g, t0s, ph, it, solver).call(init, B)
    assert rc == 0
    assert np.array_equal(out["cur"], o["cur_vals"]) and np.array_equal(out["best_vals"], o["best_vals"])
    assert np.array_equal(out["end"], o["end_spins"]) and np.array_equal(out["best"], o["best_spins"])


@pytest.mark.parametrize("n,fmt", [(20000, 1), (10000, 2)])
def test_copy_that_fits_packed_only(rfmf, ctx, oracle, n, fmt):
    # rows padded to four entries: 4 (n + 1) + 4 n entries of 2 or 4 bytes, above
    # 232,192 B beside one chain; packed 4 (n + 1) + 2 (n - 1) entries, below
    g = rfmf.random_tree(n, signed=True, seed=6)
    deg = np.diff(g.offsets.astype(np.int64))
    size = 2 if fmt == 1 else 4
    chain = 2 * n + n // 4 + 2 * 1024
    assert 4 * (n + 1) + size * int(((deg + 3) & ~3).sum()) + chain > 232192 > 4 * (n + 1) + size * int(deg.sum()) + chain
    init, solver = chains_for(g, [1, 2])
    t0s, ph, it = [100.0, 200.0], [64, 1], [10, 10]
    o = oracle.anneal(g, init, t0s, solver, ph, it)
    dg = rfmf.DeviceGraph(ctx, g)
    cfg = rfmf.make_config(csr_format=fmt, threads_per_chain=32)
    b = rfmf.Batch(ctx, [dg] * 2, t0s, solver, list(init), ph, it, cfg)
    assert b.info()["csr_format"] == (4 if fmt == 1 else 5)   # HBM walks of the entries asked for
    b.run(20)
    r = b.read()
    b.close()
    assert np.array_equal(r["cur_vals"], o["cur_vals"]) and np.array_equal(np.stack(r["end_spins"]), o["end_spins"])
    srv = rfmf.Server(ctx, window_sweeps=7, cfg=cfg)
    rid = srv.submit(dg, init[:1], t0s[:1], ph, it, solver[:1])
    assert srv.wait(rid, timeout=300)["state"] == "done"
    got = srv.result(rid)
    assert np.array_equal(got.end_spins[0], o["end_spins"][0]) and got.best_vals[0] == o["best_vals"][0]
    srv.close()
    dg.close()
