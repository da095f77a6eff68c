"""Timed cases of the annealer's public entry points.

A case is a dict of plain values; `prepare` makes what a program holds before
the call (graphs on the device, chains, a schedule), `run` is one call of the
path.  Kinds:

  anneal    one drop-in call over one graph (rfmf_anneal: host buffers in and
            out), the call a user of gpu3::annealGpu makes
  batch     chains over one or several graphs, advanced window by window or as
            CUDA-graph replays, then read back (rfmf_batch_*)
  serve     concurrent requests to a server, submitted together and awaited
  noalloc   rfmf_anneal_noalloc over the caller's own device buffers
  ingest    a graph built on the device from an edge list, and its CSR back
  output    cut values and partition strings of a finished batch

A graph is written "family size [degree]": "torus 50x60", "er 2000 19",
"tree 10000", "planar 3000" (random geometric, mean degree 11.7); several are
joined by "+".  `wmax` 0 gives weights +1, 1 gives +-1, k > 1 integers in
+-[1, k].  `phases` lists the group counts P, each run for `iters` sweeps;
t0 runs over the eight-step ladder, times `t0_scale` (weighted instances
anneal at temperatures in proportion to their weights).  Every output is a
whole number and a function of the inputs alone.
"""
import math

import numpy as np
import torch

import rfmf_gb300 as R

LADDER = [35.0, 50.0, 70.0, 100.0, 140.0, 200.0, 280.0, 400.0]
HALVING = "128,64,32,16,8,4,2,1"

_contexts = {}


def _context():
    """The program's context: one per process, as a caller keeps it."""
    if 0 not in _contexts:
        _contexts[0] = R.Context(0)
    return _contexts[0]


def _anneal(name, graphs, chains, iters, kind="anneal", wmax=1, phases=HALVING, t0_scale=1.0, **more):
    return dict(name=name, kind=kind, graphs=graphs, chains=chains, wmax=wmax, phases=phases, iters=iters,
                t0_scale=t0_scale, **more)


def listed():
    return [
        # The smallest call: a handful of short chains on a small graph, where
        # set-up, launch and read-back are the time.
        _anneal("anneal_er256_4ch", "er 256 13", 4, 64, phases="128,32,8,1"),
        # The CPU-sized configuration: G1's shape, 32 chains.
        _anneal("anneal_er800_32ch", "er 800 48", 32, 2000, wmax=0),
        # The mid-size dense graph as one drop-in call, 1024 chains.
        _anneal("anneal_er2000_1024ch", "er 2000 19", 1024, 4000),
        # The reference's own job on its largest Gset graph (G81: 100x200
        # torus), 80 chains: fewer chains than SMs.
        _anneal("anneal_torus20000_80ch", "torus 100x200", 80, 2000),
        # Integer weights: 32-bit gains and entries; group counts that are
        # not powers of two.
        _anneal("anneal_er1500_weighted", "er 1500 12", 300, 2000, wmax=1000, phases="100,60,30,12,5,1",
                t0_scale=500.0),
        # The benchmark's workload: both mid-size graphs in one batch of 2048
        # chains, advanced in windows.
        _anneal("batch_mid_2048ch", "torus 50x60+er 2000 19", 1024, 4000, kind="batch", window=8000, replays=0),
        # The large sparse configuration, 256 chains per graph.
        _anneal("batch_sparse_768ch", "torus 100x200+tree 10000+er 5000 5", 256, 1500, kind="batch", window=4000,
                replays=0),
        # Many uneven graphs side by side, as CUDA-graph replays of
        # fixed-size windows.
        _anneal("batch_many_graphs",
                "er 807 12+torus 30x41+planar 1201+er 1633 9+tree 2025+torus 50x50+planar 2999+er 3407 6+"
                "torus 60x67+tree 4801+planar 5003+er 6007 5+torus 80x90+tree 9001+planar 11003+torus 100x140",
                48, 1000, kind="batch", window=2000, replays=4),
        # Requests of uneven size that arrive together.
        _anneal("serve_8_requests", "er 5000 5+tree 7001+torus 70x100+planar 5501+er 9001 4+torus 100x120+"
                "tree 15013+torus 100x200", 0, 1024, kind="serve", window=4096),
        # A caller that owns its device memory; odd chain count and groups.
        _anneal("noalloc_planar3000_150ch", "planar 3000", 150, 1500, kind="noalloc", phases="100,30,10,3,1"),
        # Ingest of a dense random graph of half a million edge lines.
        dict(name="ingest_481k_edges", kind="ingest", n=20000, edges=481000, wmax=1),
        # Results of the 2048-chain workload: cuts and partition strings.
        _anneal("output_2048ch", "torus 50x60+er 2000 19", 1024, 25, kind="output"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, lo, hi):
    n = _log(rng, lo, hi)
    family = rng.choice(["er", "er", "torus", "tree", "planar"])
    if family == "torus":
        rows = max(3, int(math.sqrt(n) * rng.uniform(0.5, 1.0)))
        return "torus %dx%d" % (rows, max(3, n // rows))
    if family == "er":
        return "er %d %d" % (n, _log(rng, 4, min(48, max(5, n // 8))))
    return "%s %d" % (family, n)


def _draw_phases(rng):
    if rng.random() < 0.6:
        return rng.choice([HALVING, HALVING, "64,16,4,1", "32,8,2,1"])
    ps = sorted({_log(rng, 1, 200) for _ in range(rng.randint(2, 7))}, reverse=True)
    return ",".join(str(p) for p in ps)


def draw(rng):
    kind = rng.choice(["anneal"] * 9 + ["batch"] * 4 + ["serve"] * 2 + ["noalloc"] * 2 + ["ingest"] * 2 + ["output"])
    if kind == "ingest":
        n = _log(rng, 200, 30000)
        return dict(kind=kind, n=n, edges=min(480000, int(n * rng.uniform(1.1, 24.0))),
                    wmax=rng.choice([0, 1, 1, 50, 40000]))
    wmax = rng.choice([0, 1, 1, 1, 1, 5, 100, 1000])
    count = rng.randint(2, 10) if kind in ("batch", "serve") else rng.randint(1, 3) if kind == "output" else 1
    graphs = [_draw_graph(rng, 64, 20000) if kind != "serve" else _draw_graph(rng, 2000, 20000) for _ in range(count)]
    chains = _log(rng, 4, 1024 if count == 1 else 1024 // count)
    if kind == "noalloc":
        chains = _log(rng, 4, 512)
    phases = _draw_phases(rng)
    sizes = [_shape(g)[0] for g in graphs]
    # Sweeps over their logarithm, up to about a tenth of a second a pass.
    us = 3.0 + 1e-3 * max(sizes) + (128 if kind == "serve" else chains) * sum(sizes) / 5e5
    np_ = phases.count(",") + 1
    most = min(4000.0, 1e5 / us / np_)
    iters = 25 if kind == "output" else max(8, _log(rng, max(8.0, most / 32), max(16.0, most)))
    case = _anneal("", "+".join(graphs), chains, iters, kind=kind, wmax=wmax, phases=phases,
                   t0_scale=1.0 if wmax <= 5 else float(wmax) * rng.choice([0.1, 0.5, 0.5, 1.0]))
    del case["name"]
    if kind == "batch":
        replays = rng.choice([0, 0, 4])
        total = iters * np_
        case["window"] = -(-total // replays) if replays else max(1, int(total / rng.choice([1, 2, 4])))
        case["replays"] = replays
    if kind == "serve":
        case["chains"] = 0
        case["window"] = rng.choice([1024, 4096])
    return case


# ------------------------------------------------------------------ inputs
def _shape(spec):
    """(vertices, expected edges) of a graph."""
    p = spec.split()
    if p[0] == "torus":
        r, c = (int(x) for x in p[1].split("x"))
        return r * c, 2 * r * c
    n = int(p[1])
    if p[0] == "er":
        return n, int(n * float(p[2]) / 2)
    return n, (n - 1 if p[0] == "tree" else int(n * 11.7 / 2))


def _graph(spec, wmax, seed):
    p = spec.split()
    signed = wmax >= 1
    if p[0] == "torus":
        r, c = (int(x) for x in p[1].split("x"))
        g = R.torus(r, c, signed=signed, seed=seed)
    elif p[0] == "er":
        g = R.erdos_renyi_sparse(int(p[1]), float(p[2]), signed=signed, seed=seed)
    elif p[0] == "tree":
        g = R.random_tree(int(p[1]), signed=signed, seed=seed)
    else:
        g = R.planar_like(int(p[1]), signed=signed, seed=seed)
    n = _shape(spec)[0]
    if g.n < n or wmax > 1:
        # Vertices without an edge get one to the next vertex (the loader
        # would drop them), so that every seed's graph has n vertices.
        rng = np.random.default_rng(seed + 77)
        src = np.repeat(np.arange(g.n), np.diff(g.offsets.astype(np.int64)))
        up = g.col > src
        u, v, w = g.orig_ids[src[up]], g.orig_ids[g.col[up]], g.weight[up].astype(np.int64)
        lone = np.setdiff1d(np.arange(n), g.orig_ids)
        u, v = np.concatenate([u, lone]), np.concatenate([v, (lone + 1) % n])
        w = np.concatenate([w, np.ones(len(lone), np.int64)])
        if wmax > 1:
            w = rng.integers(1, wmax + 1, len(u)) * rng.choice([-1, 1], len(u))
        g = R.csr_from_edges(u, v, w)
    return g


def _edge_list(n, m, wmax, seed):
    """m edge lines over n ids of [0, 2n): a tree over all of them, random
    distinct pairs, and one line in 64 that repeats an earlier one's pair."""
    rng = np.random.default_rng(seed)
    ids = np.sort(rng.choice(2 * n, n, replace=False)).astype(np.int64)
    child = np.arange(1, n)
    key = (rng.random(n - 1) * child).astype(np.int64) * n + child
    again = m // 64
    while len(key) < m - again:
        a, b = rng.integers(0, n, m), rng.integers(0, n, m)
        more = (np.minimum(a, b) * n + np.maximum(a, b))[a != b]
        more = np.setdiff1d(more, key)
        key = np.concatenate([key, rng.permutation(more)[:m - again - len(key)]])
    key = rng.permutation(key[:m - again])
    key = np.concatenate([key, rng.choice(key, again)])
    u, v = key // n, key % n
    flip = rng.random(m) < 0.5
    w = rng.integers(1, max(1, wmax) + 1, m)
    if wmax:
        w = w * rng.choice([-1, 1], m)
    return ids[np.where(flip, v, u)], ids[np.where(flip, u, v)], w.astype(np.int64)


def _chains(n, count, case, first):
    """Initial spins, t0s and solver seeds of `count` chains with raw seeds first, first + 1, ..."""
    seeds = range(first, first + count)
    init = np.stack([R.initial_spins(s, n) for s in seeds])
    t0s = [LADDER[c % 8] * case["t0_scale"] for c in range(count)]
    return init, t0s, [R.solver_seed(s) for s in seeds]


def _request_chains(k):
    """Chains of a served request: 16 to 256, uneven."""
    return [16, 256, 48, 128, 33, 96, 64, 20][k % 8]


def prepare(case, seed):
    kind = case["kind"]
    ctx = _context()
    if kind == "ingest":
        u, v, w = _edge_list(case["n"], case["edges"], case["wmax"], seed)
        return dict(case=case, ctx=ctx, u=u, v=v, w=w)
    phases = [int(x) for x in case["phases"].split(",")]
    st = dict(case=case, ctx=ctx, phases=phases, iters=[case["iters"]] * len(phases))
    graphs = [_graph(s, case["wmax"], seed * 31 + k) for k, s in enumerate(case["graphs"].split("+"))]
    st["graphs"] = graphs
    first = (seed % 1000003) * 4096
    if kind == "noalloc":
        _prepare_noalloc(st, graphs[0], first)
        return st
    st["dgs"] = [R.DeviceGraph(ctx, g) for g in graphs]
    counts = [_request_chains(k) if kind == "serve" else case["chains"] for k in range(len(graphs))]
    st["sets"] = [_chains(g.n, c, case, first + 512 * k) for k, (g, c) in enumerate(zip(graphs, counts))]
    if kind == "serve":
        st["server"] = R.Server(ctx, window_sweeps=case["window"])
    if kind == "output":
        st["batch"] = _batch(st)
        st["batch"].run(sum(st["iters"]))
        st["stride"] = max(g.n for g in graphs)
        st["text"] = np.zeros((st["batch"].C, st["stride"]), np.uint8)
    return st


def _prepare_noalloc(st, g, first):
    case, dev = st["case"], torch.device("cuda", 0)
    init, t0s, solver = _chains(g.n, case["chains"], case, first)
    end, val, off = R.beta_tables(t0s, sum(st["iters"]))
    starts = sorted(set(off.tolist())) + [len(end)]
    runs = {s: starts[i + 1] - s for i, s in enumerate(starts[:-1])}
    words = (g.n + 31) // 32
    bits = np.packbits(np.pad(init > 0, ((0, 0), (0, 32 * words - g.n))), axis=1, bitorder="little")
    st.update(
        off=torch.from_numpy(g.offsets.astype(np.int32)).to(dev),
        edges=torch.from_numpy(np.stack([g.col, g.weight], 1).astype(np.int32).ravel()).to(dev),
        end=torch.from_numpy(end).to(dev), val=torch.from_numpy(val).to(dev),
        start=torch.from_numpy(bits.view(np.int32).copy()).to(dev),
        t0s=np.array(t0s, np.float64), solver=np.array(solver, np.uint64), B=g.max_weighted_degree(),
        chain_off=off, chain_runs=np.array([runs[int(o)] for o in off], np.int64),
        ph=np.array(st["phases"], np.uint64), it=np.array(st["iters"], np.uint64))


def _batch(st):
    gl, t0s, sol, ini = [], [], [], []
    for dg, (init, t, s) in zip(st["dgs"], st["sets"]):
        gl += [dg] * len(t)
        t0s += t
        sol += s
        ini += list(init)
    return R.Batch(st["ctx"], gl, t0s, sol, ini, st["phases"], st["iters"])


# --------------------------------------------------------------- one pass
def _results(r):
    return dict(end=r.end_spins, best=r.best_spins, best_vals=r.best_vals, final_vals=r.final_vals)


def run(st):
    return {"anneal": _run_anneal, "batch": _run_batch, "serve": _run_serve, "noalloc": _run_noalloc,
            "ingest": _run_ingest, "output": _run_output}[st["case"]["kind"]](st)


def _run_anneal(st):
    init, t0s, sol = st["sets"][0]
    return _results(R.anneal_gpu(st["ctx"], st["dgs"][0], st["graphs"][0].max_weighted_degree(), init, t0s,
                                 st["phases"], st["iters"], sol))


def _run_batch(st):
    case, total = st["case"], sum(st["iters"])
    b = _batch(st)
    if case["replays"]:
        b.run_graph(case["window"], launches=1, replays=case["replays"])
    else:
        for done in range(0, total, case["window"]):
            b.run(min(case["window"], total - done))
    r = b.read()
    b.close()
    return dict(end=np.concatenate(r["end_spins"]), best=np.concatenate(r["best_spins"]), cur=r["cur_vals"],
                best_vals=r["best_vals"], done=r["sweeps_done"].astype(np.int64))


def _run_serve(st):
    srv = st["server"]
    ids = [srv.submit(dg, init, t, st["phases"], st["iters"], s) for dg, (init, t, s) in zip(st["dgs"], st["sets"])]
    for rid in ids:
        srv.wait(rid)
    return [_results(srv.result(rid)) for rid in ids]


def _run_noalloc(st):
    bits = st["start"].clone()
    best_bits = torch.empty_like(bits)
    C = bits.shape[0]
    cur = torch.empty(C, dtype=torch.int64, device=bits.device)
    best = torch.empty(C, dtype=torch.int64, device=bits.device)
    L = R.lib()
    rc = L.rfmf_anneal_noalloc(
        0, None, st["graphs"][0].n, st["off"].data_ptr(), st["edges"].data_ptr(), st["B"], C,
        st["t0s"].ctypes.data, st["solver"].ctypes.data, len(st["ph"]), st["ph"].ctypes.data, st["it"].ctypes.data,
        st["end"].data_ptr(), st["val"].data_ptr(), st["end"].numel(), st["chain_off"].ctypes.data,
        st["chain_runs"].ctypes.data, bits.data_ptr(), best_bits.data_ptr(), cur.data_ptr(), best.data_ptr())
    if rc:
        raise RuntimeError("rfmf_anneal_noalloc: %s" % L.rfmf_last_error().decode())
    return dict(end=bits, best=best_bits, cur=cur, best_vals=best)


def _run_ingest(st):
    g = R.DeviceGraph.from_edges(st["ctx"], st["u"], st["v"], st["w"])
    off, col, w = g.csr()
    out = dict(offsets=off.view(np.int32), col=col, weight=w, ids=g.orig_ids(), **g.info())
    g.close()
    return out


def _run_output(st):
    b, text = st["batch"], st["text"]
    end, best = b.cuts(), b.cuts(best=True)
    rc = R.lib().rfmf_batch_partitions(b.h, 1, text.ctypes.data, st["stride"])
    if rc:
        raise RuntimeError("rfmf_batch_partitions: %s" % R.lib().rfmf_last_error().decode())
    return dict(end_cuts=end, best_cuts=best, text=text)


# ------------------------------------------------------------------- work
def work(case):
    """Bytes: inputs read once (graph, spins, records), outputs written once.
    `flops` counts integer operations: per sweep and block of eight vertices
    Philox4x32-10 (10 rounds of two wide multiplies and four xors), four per
    vertex for its key, and four per entry of the winners' rows."""
    if case["kind"] == "ingest":
        n, m = case["n"], case["edges"]
        return {"bytes": 24 * m + 2 * m * 8 + 12 * n, "flops": 8 * m}
    sched = [(int(p), case["iters"]) for p in case["phases"].split(",")]
    nbytes = flops = 0.0
    for k, spec in enumerate(case["graphs"].split("+")):
        n, m = _shape(spec)
        C = _request_chains(k) if case["kind"] == "serve" else case["chains"]
        nbytes += 4 * n + 16 * m
        if case["kind"] == "output":
            nbytes += C * (n + 2 * n / 8 + 16)
            flops += C * 4 * 2 * m
            continue
        nbytes += C * (3 * n + 40)
        for P, it in sched:
            flops += C * it * (n * (60 / 8 + 4) + 4 * min(P, n) * 2 * m / n)
    return {"bytes": nbytes, "flops": flops}


def exact(case, seed):
    """No output is a rounded number: all are integers, the same bit for bit."""
    return None
