"""The device record of a graph (device_graph, rfmf_gb300/csrc/rfmf_host.h),
compiled into a small harness with g++ (host only).  A server keeps one record
per graph for requests of any CSR format, so what a staging kernel copies (row
words and the entries of its width) must be the csr_bytes its CTA keeps room
for, and no entry array a graph has may be missing, whatever format the record
was first made for."""
import shutil
import subprocess

import pytest

from conftest import ROOT
from test_host_helpers import _cuda_include

RECORD = r"""
#include <cstdio>
#include "rfmf_host.h"
int rfmf::fail(int c, const char*, ...) { return c; }
void rfmf::let_go(rfmf_context*) {}
void rfmf::let_go(const rfmf_graph*) {}
extern "C" cudaError_t cudaFree(void*) { return cudaSuccess; }
using namespace rfmf;
int main() {
    static char u16, p32, edges;
    static uint32_t offsets[2 * 56016 / 4];   // row words behind the offsets
    for (int has = 1; has < 4; ++has) {   // 16-bit entries, 32-bit entries, both
        auto* g = new rfmf_graph();
        g->n = 14000;
        g->rowBytes = 56016;
        g->offsets.p = offsets;
        g->edges.p = &edges;
        if (has & 1) { g->unit16 = true; g->u16Bytes = 111984; g->u16.p = &u16; }
        if (has & 2) { g->packed32 = true; g->p32Bytes = 223968; g->p32.p = &p32; }
        const DevGraph d = device_graph(g);
        if (has & 1)
            if (static_cast<const void*>(d.u16) != &u16 || d.rowBytes + d.u16Bytes != csr_bytes(g, kCsrUnit16)) return 1;
        if (has & 2)
            if (static_cast<const void*>(d.p32) != &p32 || d.rowBytes + d.p32Bytes != csr_bytes(g, kCsrPacked32)) return 2;
        if (d.offsets != offsets || d.rows != offsets + 56016 / 4 || static_cast<const void*>(d.edges) != &edges) return 3;
    }
    puts("ok");
    return 0;
}
"""


def test_record_serves_every_format(tmp_path):
    cxx, inc = shutil.which("g++"), _cuda_include()
    if not cxx or not inc:
        pytest.skip("g++ or the CUDA headers are missing")
    src, exe = tmp_path / "record.cpp", tmp_path / "record"
    src.write_text(RECORD)
    subprocess.run([cxx, "-O1", "-std=c++17", "-Wall", "-I", str(ROOT / "rfmf_gb300" / "csrc"), "-I", inc, str(src),
                    "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.returncode
