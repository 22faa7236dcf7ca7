"""The FP64 flux at the edges of its number range: its reciprocals against long double, NaN neighbours and
overflowing gradients."""
import os
import shutil
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import cdd
import cdd_oracle as O

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "cuda-plasticity_b200", "csrc")

PROG = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "fp64_math.cuh"
__global__ void both(const double* x, double* r, double* s, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { s[i] = cdd::rsqrt_f64(x[i]); r[i] = cdd::rcp_f64(x[i]); }
}
int main() {
    std::mt19937_64 g(1);
    std::uniform_real_distribution<double> man(1.0, 2.0), ex(-300.0, 300.0);
    std::vector<double> x = {0.0, INFINITY, -1.0, NAN, 1.0, 4.0, 2.0};
    for (int e = -1022; e <= 1021; ++e) { x.push_back(std::ldexp(1.0, e)); x.push_back(std::ldexp(2.0 - 0x1p-52, e)); }
    const int edge = (int)x.size();
    for (int i = 0; i < 2000000; ++i) x.push_back(std::ldexp(man(g), (int)ex(g)));
    const int n = (int)x.size();
    double *dx, *dr, *ds;
    if (cudaMalloc(&dx, 8 * n) || cudaMalloc(&dr, 8 * n) || cudaMalloc(&ds, 8 * n)) return 2;
    std::vector<double> r(n), s(n);
    cudaMemcpy(dx, x.data(), 8 * n, cudaMemcpyHostToDevice);
    both<<<(n + 255) / 256, 256>>>(dx, dr, ds, n);
    cudaMemcpy(r.data(), dr, 8 * n, cudaMemcpyDeviceToHost);
    if (cudaMemcpy(s.data(), ds, 8 * n, cudaMemcpyDeviceToHost)) return 3;
    const bool special = std::isinf(s[0]) && s[0] > 0 && std::isinf(r[0]) && s[1] == 0 && r[1] == 0 && std::isnan(s[2]) && r[2] == -1.0 &&
                         std::isnan(s[3]) && std::isnan(r[3]) && r[4] == 1.0 && s[4] == 1.0 && r[5] == 0.25 && s[5] == 0.5;
    long double er = 0, es = 0;
    for (int i = 4; i < n; ++i) {
        er = std::fmax(er, std::fabs((long double)r[i] * x[i] - 1.0L));
        const long double want = 1.0L / std::sqrt((long double)x[i]);
        es = std::fmax(es, std::fabs((long double)s[i] / want - 1.0L));
    }
    std::printf("%d %d %.6Lg %.6Lg\n", edge, (int)special, er * 0x1p52L, es * 0x1p52L);
    return 0;
}
"""


def test_reciprocals_against_long_double(tmp_path):
    """Relative error below 2^-52 over the normal range (half an ulp for the last operation, at most as much for the
    residual's rounding), and the values of 0, infinity, negative numbers and NaN."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is missing")
    src, exe = tmp_path / "math.cu", tmp_path / "math"
    src.write_text(PROG)
    r = subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC, str(src),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()
    assert int(out[1]) == 1
    assert float(out[2]) < 1.0 and float(out[3]) < 1.0, out


@pytest.mark.parametrize("shape,at", [((16, 40), (7, 20)), ((8, 12, 72), (3, 5, 40)), ((8, 6, 18), (0, 1, 0))])
def test_nan_reaches_the_nearest_cells_only(shape, at, monkeypatch):
    """A NaN two cells away leaves the limited derivative at its difference, whatever the NaN's sign bit: every cell
    that is not the NaN's own or its nearest neighbour along an axis has the finite value of a limiter that takes
    no part of it (FP64 1e-12 as for the other fluxes)."""
    minmod3 = O.minmod3
    monkeypatch.setattr(O, "minmod3", lambda a, b, c: np.where(np.isnan(a) | np.isnan(c), 0.0,
                                                               minmod3(*(np.nan_to_num(v) for v in (a, b, c)))))
    b = cdd.gaussian_random_field(shape, 0.08, 0.05, 13)
    plan = cdd.Plan([cdd.Instance(shape)], "f64")
    sigma = plan.stress(plan.pack([b]))
    far = np.ones(shape, bool)
    for d in range(len(shape)):
        for k in (-1, 0, 1):
            far[at[:d] + ((at[d] + k) % shape[d],) + at[d + 1:]] = False
    total = O.stress(b, 1.0, 0.3)
    for sign in (1.0, -1.0):
        bad = b.copy()
        bad[(4,) + at] = np.copysign(np.nan, sign)
        rhs, speed = plan.flux(plan.pack([bad]), 0.0, sigma=sigma)
        ref, ref_speed = O.flux(bad, total)
        got, got_speed = plan.field_view(rhs, 0).cpu().numpy(), speed.cpu().numpy().reshape(shape)
        assert np.isnan(got_speed[at]) and np.isfinite(got[:, far]).all()
        assert np.linalg.norm(got[:, far] - ref[:, far]) < 1e-12 * np.linalg.norm(ref[:, far])
        assert np.linalg.norm(got_speed[far] - ref_speed[far]) < 1e-12 * np.linalg.norm(ref_speed[far])


def test_overflowing_gradients_stand_still():
    """|rho|^2 past the range makes 1/|rho| zero: no velocity, no flux, and the least speed (ME per axis)."""
    shape = (12, 40)
    b = np.zeros((9,) + shape)
    b[8] = np.random.default_rng(1).standard_normal(shape) * 1e160
    plan = cdd.Plan([cdd.Instance(shape)], "f64")
    sigma = torch.ones(plan.stress_elems, dtype=torch.float64, device="cuda")
    rhs, speed = plan.flux(plan.pack([b]), 0.0, sigma=sigma)
    assert (rhs == 0).all() and torch.equal(speed, torch.full_like(speed, 2 * 2.0 ** -52))
