"""Cuts of small and mixed batches: graphs at the edges of a row slice (256 rows)
and of the size whose CTAs share a launch (4,096 vertices), groups of one to 33
chains, alone and together, against the host's cut of the spins read back; and
the rule that splits a graph's rows (host only)."""
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT, chains_for
from test_host_helpers import _cuda_include

SIZES = [(64, 33), (255, 1), (256, 31), (257, 32), (513, 33), (4096, 5), (4097, 5)]


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [SIZES] + [[s] for s in SIZES], ids=lambda s: "all" if len(s) > 1 else str(s[0]))
def test_cuts_match_spins(rfmf, ctx, sizes):
    dgs, gl, graphs, init, solver = [], [], [], [], []
    for k, (n, C) in enumerate(sizes):
        g = rfmf.random_tree(n, signed=True, seed=n)
        g.weight = g.weight * (k + 1)
        i, s = chains_for(g, list(range(100 * k, 100 * k + C)))
        dgs.append(rfmf.DeviceGraph(ctx, g))
        gl += [dgs[-1]] * C
        graphs += [g] * C
        init += list(i)
        solver += s
    b = rfmf.Batch(ctx, gl, [60.0] * len(gl), solver, init, [4, 1], [20, 20])
    for sweeps in (15, 25):   # the items are laid out at the first call, for all later ones
        b.run(sweeps)
        for best in (False, True):
            got = b.cuts(best=best)
            spins = b.read()["best_spins" if best else "end_spins"]
            assert got.tolist() == [rfmf.cut_value(g, s) for g, s in zip(graphs, spins)]
    b.close()
    for dg in dgs:
        dg.close()


RULE = r"""
#include <cstdio>
#include "rfmf_host.h"
using namespace rfmf;
int main() {
    for (int64_t n : {1, 64, 256, 257, 700, 3000, 20000, 1000000})
        for (int64_t groups : {1, 2, 64, 609, 100000}) {
            const int s = cut_slices(n, groups, 152);
            if (s < 1 || s > 64) return 1;
            if (s > 1 && n / s < 128) return 2;              // never a CTA for a few rows
            if (s > 1 && (s - 1) * groups >= 608) return 3;  // nor more CTAs than fill the SMs
        }
    if (cut_slices(64, 1, 152) != 1 || cut_slices(20000, 1, 152) != 64) return 4;
    puts("ok");
    return 0;
}
"""


def test_slice_rule(tmp_path):
    cxx, inc = shutil.which("g++"), _cuda_include()
    if not cxx or not inc:
        pytest.skip("g++ or the CUDA headers are missing")
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text(RULE)
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", str(ROOT / "rfmf_gb300" / "csrc"), "-I", inc, str(src), "-o", str(exe)],
                   check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.returncode
