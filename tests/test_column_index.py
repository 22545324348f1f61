"""W from the column index where the index nearly fills 32 bits: the kernel's own code
(w_by_columns) compiled for the CPU and run thread by thread on one column that ends just
below 2^32, which no test could allocate.  Every rank of the column takes its word once,
and nothing outside it is read."""
import os
import shutil
import subprocess
import tempfile

import pytest

from conftest import ROOT

MAIN = r"""
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>
#define __device__
#define __forceinline__ inline
#define __restrict__
struct Dim { unsigned x; };
static Dim threadIdx, blockIdx, blockDim, gridDim;
static const unsigned *lo, *hi;
static unsigned __ldg(const unsigned *p) {
    if (p < lo || p >= hi) {
        std::printf("read %td entries from the column\n", p - lo);
        std::exit(1);
    }
    return *p;
}
static void atomicXor(unsigned long long *p, unsigned long long v) { *p ^= v; }
constexpr int kGStride = 2;
#include "w_by_columns.inc"
int main() {
    for (unsigned len : {1u, 33u, 100u, 200000u}) {
        const unsigned end = 0xfffffffeu;  // the largest index of a column's end
        std::vector<unsigned> column(len), start = {end - len, end};
        for (unsigned i = 0; i < len; i++) column[i] = i;
        lo = column.data();
        hi = lo + len;
        const int32_t nz = 0;
        const uint64_t T[2] = {5, 9};
        std::vector<uint64_t> W0(len), W1(len);
        Columns co;
        co.start = start.data();
        co.ranks = reinterpret_cast<const unsigned *>(reinterpret_cast<uintptr_t>(lo) - 4ull * (end - len));
        co.nz = &nz;
        co.segs = 1;
        co.seg_shift = 30;
        blockDim.x = 1024;
        gridDim.x = 152;
        for (blockIdx.x = 0; blockIdx.x < gridDim.x; blockIdx.x++)
            for (threadIdx.x = 0; threadIdx.x < blockDim.x; threadIdx.x++)
                w_by_columns<2>(co, T, 1u, (long long)len, W0.data(), W1.data(), nullptr);
        for (unsigned i = 0; i < len; i++)
            if (W0[i] != 5 || W1[i] != 9) {
                std::printf("rank %u of %u: %llu %llu\n", i, len, (unsigned long long)W0[i], (unsigned long long)W1[i]);
                return 1;
            }
    }
    std::puts("ok");
}
"""


def test_a_column_that_ends_at_the_last_index():
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    text = open(os.path.join(ROOT, "minimumcyclebasis_gb300", "csrc", "gpu", "mcbgpu_solver.cu")).read()
    begin = text.index("struct Columns {")
    code = text[begin:text.index("\n}\n", text.index("w_by_columns(", begin)) + 3]
    with tempfile.TemporaryDirectory() as d:
        open(os.path.join(d, "w_by_columns.inc"), "w").write(code)
        src, exe = os.path.join(d, "main.cpp"), os.path.join(d, "main")
        open(src, "w").write(MAIN)
        subprocess.run([gxx, "-std=c++17", "-O1", "-I" + d, "-o", exe, src], check=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
