"""Every FFT length with a two-pass form (and some without) on each axis of the stress solve, against the CPU
oracle; the solve's adjoint by the dot-product identity; column and line tilings bitwise.

Tolerances: FP64 1e-12 rel-L2 as for the other shapes, FP32 2e-6 (as for the plane waves), the dot-product
identity 1e-12 of the product of the norms (FP64).
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import cdd
import cdd_oracle as O

SYM = [0, 1, 2, 4, 5, 8]
LENGTHS = [6, 10, 12, 16, 18, 20, 24, 36, 40, 48, 50, 54, 64, 72, 80, 96, 100, 108, 128, 144, 160, 162, 192, 200, 216, 250,
           256, 288, 320, 324, 384, 400, 432, 486, 500, 512, 640, 768, 864, 1000, 1024]


def field(shape, seed):
    return np.random.default_rng(seed).standard_normal((9,) + shape) * 0.05


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("n", LENGTHS)
def test_stress_of_every_length_against_oracle(n):
    shapes = [(n, 8), (8, n), (4, n, 6), (n, 4, 6), (6, 4, n)]
    fields = [field(s, n + i) for i, s in enumerate(shapes)]
    for prec, tol in (("f64", 1e-12), ("f32", 2e-6)):
        for shape, b in zip(shapes, fields):
            if prec == "f32":
                b = b.astype(np.float32).astype(np.float64)
            plan = cdd.Plan([cdd.Instance(shape, mu=1.3, nu=0.28)], prec)
            got = plan.stress_view(plan.stress(plan.pack([b])), 0).cpu().numpy()
            assert rel(got, O.stress(b, 1.3, 0.28)[SYM]) < tol, (shape, prec)
            plan.close()


@pytest.mark.parametrize("shape", [(24, 18, 20), (50, 12), (36, 100, 48), (16, 162, 250)])
def test_stress_adjoint_dot_product(shape):
    plan = cdd.Plan([cdd.Instance(shape)], "f64")
    b = plan.pack([field(shape, 1)])
    s = plan.stress(b)
    y = torch.randn(plan.stress_elems, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    back = plan.empty_field()
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    assert plan.lib.cdd_stress_adjoint(plan.handle, ptr(y), ptr(back), ctypes.c_void_p(0)) == 0
    torch.cuda.synchronize()
    left, right = float(torch.dot(s, y)), float(torch.dot(b, back))
    assert abs(left - right) < 1e-12 * float(s.norm() * y.norm())


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_tilings_change_no_bit(prec):
    shape = (36, 54, 40)
    b = field(shape, 3)
    want = None
    for t in ({}, {"green_cols": 1}, {"green_cols": 8}, {"mid_cols": 1}, {"mid_cols": 4}, {"rows_lines": 1}, {"rows_lines": 7}):
        plan = cdd.Plan([cdd.Instance(shape)], prec, tuning=[t] if t else None)
        s = plan.stress(plan.pack([b]))
        want = s if want is None else want
        assert torch.equal(s, want), t
