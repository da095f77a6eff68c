"""The host check of a CSR (rfmf_csr_validate, rfmf_graph_create; no GPU): small
random graphs, valid and with one or two things wrong, against the invariants
spelled out; what is first wrong is named as before."""
import ctypes as ct

import numpy as np
import pytest


def _expected(n, off, col, w):
    """(status, message) of the first violation in row order, or (0, B)."""
    B = 0
    for v in range(n):
        if off[v + 1] < off[v]:
            return 1, f"offsets not monotone at {v}"
        s = 0
        for i in range(off[v], off[v + 1]):
            u = int(col[i])
            if not 0 <= u < n:
                return 1, f"col[{i}]={u} out of range"
            if u == v:
                return 1, f"self loop at vertex {v}"
            if i > off[v] and col[i - 1] >= u:
                return 1, f"row {v} not strictly ascending"
            if w[i] == 0:
                return 1, f"zero weight on edge ({v},{u})"
            if off[u + 1] < off[u]:
                return 1, f"offsets not monotone at {u}"
            # a binary search of row u for v, as the check does one
            lo, hi = int(off[u]), int(off[u + 1])
            while lo < hi:
                mid = lo + (hi - lo) // 2
                if col[mid] < v:
                    lo = mid + 1
                else:
                    hi = mid
            if lo == off[u + 1] or col[lo] != v or w[lo] != w[i]:
                return 1, f"edge ({v},{u}) has no symmetric twin"
            s += abs(int(w[i]))
        B = max(B, s)
    return 0, B


def _check(rfmf, n, off, col, w):
    off, col, w = (np.ascontiguousarray(off, np.uint32), np.ascontiguousarray(col, np.int32),
                   np.ascontiguousarray(w, np.int32))
    B = ct.c_int64(-1)
    rc = rfmf.lib().rfmf_csr_validate(n, off.ctypes.data, col.ctypes.data, w.ctypes.data, ct.byref(B))
    return rc, B.value if rc == 0 else rfmf.lib().rfmf_last_error().decode()


@pytest.mark.parametrize("seed", range(4))
def test_random_graphs_and_faults(rfmf, seed):
    rng = np.random.default_rng(seed)
    bad = 0
    for _ in range(400):
        n = int(rng.integers(1, 12))
        adj = {}
        for a in range(n):
            for b in range(a + 1, n):
                if rng.random() < 0.4:
                    adj[a, b] = adj[b, a] = int(rng.integers(1, 5)) * (1 if rng.random() < 0.5 else -1)
        keys = sorted(adj)
        off = np.searchsorted([k[0] for k in keys] or [], np.arange(n + 1)).astype(np.int64)
        col = np.array([k[1] for k in keys], np.int64)
        w = np.array([adj[k] for k in keys], np.int64)
        for _ in range(int(rng.integers(0, 3))):
            if not len(col):
                break
            i = int(rng.integers(0, len(col)))
            kind = rng.integers(0, 4)
            if kind == 0:
                col[i] = rng.integers(-1, n + 1)
            elif kind == 1:
                w[i] = rng.integers(-2, 3)
            elif kind == 2 and n > 2:
                off[int(rng.integers(1, n))] = rng.integers(0, len(col) + 1)
            else:
                j = int(rng.integers(0, len(col)))
                col[i], col[j] = col[j], col[i]
        want, got = _expected(n, off, col, w), _check(rfmf, n, off, col, w)
        bad += want[0]
        assert got == want, (n, off.tolist(), col.tolist(), w.tolist())
    assert 50 < bad < 390
