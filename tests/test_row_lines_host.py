"""Shared memory of the row passes over every length, largest radix, precision and line count that a plan takes:
a host program built by nvcc from csrc/cdd_internal.cuh (no CUDA calls). A count that the two line buffers fit
(with dense twiddle rows: the rule that accepts a launch shape) must fit in the form that rows_fit leaves."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "cuda-plasticity_b200", "csrc")

PROG = r"""
#include <cstdio>
#include <cstring>
#include "cdd_internal.cuh"
using namespace cdd;
static bool line_plan(int n, int e, LinePlan& lp, size_t velt) {
    std::memset(&lp, 0, sizeof lp);
    int m = n, a = 0, st = 0, ns = 1;
    while (m % 2 == 0) { m /= 2; ++a; }
    int q = a / e, rest = a % e;
    const bool fold = rest == 1 && q > 0 && e >= 3;
    for (int i = 0; i < q - fold; ++i) lp.radix[st++] = 1 << e;
    if (fold) { lp.radix[st++] = 1 << (e - 1); lp.radix[st++] = 4; }
    else if (rest) lp.radix[st++] = 1 << rest;
    for (int p : {3, 5}) while (m % p == 0) { m /= p; lp.radix[st++] = p; }
    if (m != 1 || a < 1 || (n % 3 == 0 && n % 5 == 0)) return false;
    lp.n = n; lp.nst = st;
    for (int i = 0; i < st; ++i) { lp.nr[i] = fdiv_make(n / lp.radix[i]); lp.ns[i] = fdiv_make(ns); ns *= lp.radix[i]; }
    set_two_pass(lp);
    std::vector<double> re(n, 1.0), im(n, 0.0);
    append_stage_twiddles(lp, re, im, velt);
    return true;
}
int main() {
    const size_t optin = 232448;
    long long shapes = 0, bad = 0, engine = 0;
    for (int n = 4; n <= 1024; n += 2)
        for (int e = 2; e <= 4; ++e)
            for (int velt = 8; velt <= 16; velt += 8) {
                LinePlan lp;
                if (!line_plan(n, e, lp, velt)) continue;
                for (int P = 1; P <= 1024; ++P) {
                    const size_t dense = (((size_t)(rows_io_plan(lp, P) ? 1 : 2) * P * (n + (n >> 4) + 1) + 1) & ~(size_t)1) * velt +
                                         (size_t)lp.twvalues * velt + rows_table_bytes(P);
                    if (dense + 1024 > optin) continue;
                    LinePlan own = lp;
                    rows_fit(own, P, velt, optin - 1024);
                    ++shapes;
                    engine += own.pa != lp.pa;
                    bad += rows_smem_bytes(own, P, velt) > optin;
                }
            }
    std::printf("%lld %lld %lld\n", shapes, engine, bad);
    return 0;
}
"""


def test_every_accepted_row_shape_fits(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is missing")
    src, exe = tmp_path / "rows.cu", tmp_path / "rows"
    src.write_text(PROG)
    r = subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                        "--expt-relaxed-constexpr", "-I", CSRC, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    shapes, engine, bad = map(int, subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    assert shapes > 10_000 and engine > 0 and bad == 0
