"""Launch shapes of plans with several instances: the lines per block of the row passes come from the plan's
whole work, and an instance's results do not depend on what it shares its plan with."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import cdd
import cdd_oracle as O


@pytest.mark.parametrize("prec,full", [("f64", 2048), ("f32", 4096)])
def test_row_lines_come_from_the_whole_plan(prec, full):
    """64 grids together take lines for about four blocks per SM, or whole blocks, where one such grid alone takes
    single lines (results: the oracle tests)."""
    shapes = [(96, 96), (100, 100)] * 32
    plan = cdd.Plan([cdd.Instance(s) for s in shapes], prec)
    lines = [plan.tuning(i)["rows_lines"] for i in range(len(shapes))]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert all(n == full // s[1] for n, s in zip(lines, shapes)) or sum(3 * s[0] / n for n, s in zip(lines, shapes)) < 4.4 * sms
    assert cdd.Plan([cdd.Instance(shapes[0])], prec).tuning(0)["rows_lines"] == 1


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(4, 32), (6, 32), (4, 6, 64), (10, 128), (18, 50), (24, 24, 24)])
def test_stress_of_an_instance_does_not_depend_on_its_batch(shape, prec):
    b = [cdd.gaussian_random_field(s, 0.1, 0.05, 5 + i) for i, s in enumerate([shape, (96, 96), (100, 100)])]
    one = cdd.Plan([cdd.Instance(shape)], prec)
    want = one.stress(one.pack(b[:1]))
    many = cdd.Plan([cdd.Instance(x.shape[1:]) for x in [b[0]] + b[1:] * 32], prec)
    got = many.stress(many.pack([b[0]] + b[1:] * 32))
    assert torch.equal(many.stress_view(got, 0), one.stress_view(want, 0))


@pytest.mark.parametrize("lines", [829, 830, 850, 903])
def test_largest_row_lines_of_a_ten_point_axis_run(lines):
    """FP32 line counts that fit two line buffers but not the (larger) two-pass form of 10 points (FP32 2e-6
    rel-L2 as for the other lengths)."""
    b = np.random.default_rng(3).standard_normal((9, 320, 10)) * 0.05
    plan = cdd.Plan([cdd.Instance((320, 10))], "f32", tuning=[{"rows_lines": lines}])
    assert plan.tuning(0)["rows_lines"] == lines
    got = plan.stress_view(plan.stress(plan.pack([b])), 0).cpu().numpy()
    want = O.stress(b.astype(np.float32).astype(np.float64), 1.0, 0.3)[[0, 1, 2, 4, 5, 8]]
    assert np.linalg.norm(got - want) < 2e-6 * np.linalg.norm(want)


def test_row_lines_past_the_shared_memory_are_refused():
    with pytest.raises(cdd.CDDError) as e:
        cdd.Plan([cdd.Instance((320, 10))], "f32", tuning=[{"rows_lines": 920}])
    assert e.value.code == 1


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_a_plan_of_every_fft_form(prec):
    """One plan whose axes take one-stage passes, passes of up to 16 and of more values, and lengths without a two-pass
    form: each instance has the stress, its adjoint and the observables of its own plan."""
    shapes = [(64, 64, 8), (36, 54, 8), (100, 20, 8), (20, 100, 8), (288, 6, 8), (6, 288, 8), (512, 4, 8), (4, 4, 4)]
    fields = [np.random.default_rng(i).standard_normal((9,) + s) * 0.05 for i, s in enumerate(shapes)]
    many = cdd.Plan([cdd.Instance(s) for s in shapes], prec)

    def results(plan, b):
        beta = plan.pack(b)
        sig = plan.stress(beta)
        back = plan.empty_field()
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())
        assert plan.lib.cdd_stress_adjoint(plan.handle, ptr(sig), ptr(back), ctypes.c_void_p(0)) == 0
        return sig, back, plan.observe("rho", beta), plan.observe("rotation", beta)

    got = results(many, fields)
    for i, s in enumerate(shapes):
        one = cdd.Plan([cdd.Instance(s)], prec)
        want = results(one, [fields[i]])
        views = (many.stress_view(got[0], i), many.field_view(got[1], i), many.observable_view(got[2], i, "rho"),
                 many.observable_view(got[3], i, "rotation"))
        for a, w in zip(views, want):
            assert torch.equal(a.reshape(-1), w), s
