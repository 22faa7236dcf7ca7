"""The time step set by stage 1's last block in plans of several instances, and plan kernels that follow other work
through an event."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import cdd


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_a_nonfinite_instance_stops_alone(prec, graph):
    """The other instances of the plan step as they do alone, the stopped one keeps its field and time, and after its
    field is made finite the same plan steps it too (every count of finished blocks went back to zero)."""
    shapes = [(32, 32, 32), (16, 48), (24, 24, 24)]
    insts = [cdd.Instance(s, load_rate=(-0.025, -0.025, 0.05)) for s in shapes]
    good = [cdd.gaussian_random_field(s, 0.06, 0.05, 40 + i) for i, s in enumerate(shapes)]
    bad = good[1].copy()
    bad[4, 3, 7] = np.nan
    plan = cdd.Plan(insts, prec)
    beta = plan.pack([good[0], bad, good[2]])
    plan.set_time(0.0, 1e30)
    plan.run(beta, 2, graph=graph)
    with pytest.raises(cdd.CDDError) as e:
        plan.check_status()
    assert e.value.code == 4
    t, _, active = plan.get_time()
    assert list(active) == [True, False, True] and t[1] == 0.0
    assert torch.equal(plan.field_view(beta, 1).nan_to_num(nan=7.0), torch.as_tensor(bad, device="cuda").to(plan.dtype).nan_to_num(nan=7.0))
    plan.field_view(beta, 1).copy_(torch.as_tensor(good[1]))
    plan.run(beta, 1, graph=graph)
    plan.check_status()
    for i, steps in enumerate((3, 1, 3)):
        one = cdd.Plan([insts[i]], prec)
        alone = one.pack([good[i]])
        one.set_time(0.0, 1e30)
        one.run(alone, steps, graph=graph)
        assert torch.equal(plan.field_view(beta, i).reshape(-1), alone)
        assert plan.get_time()[0][i] == one.get_time()[0][0]


def work(dst, src, k, reps):
    """dst = k src after `reps` passes over a larger buffer, so that the copy comes late."""
    big = torch.zeros(1 << 24, device="cuda")
    for _ in range(reps):
        big.add_(1.0)
    torch.mul(src, k, out=dst)


def test_kernels_after_an_event_see_the_other_streams_work():
    shape = (32, 24, 32)
    plan = cdd.Plan([cdd.Instance(shape)], "f64")
    src = plan.pack([cdd.gaussian_random_field(shape, 0.06, 0.05, 3)])
    beta, out, rhs = torch.zeros_like(src), plan.empty_stress(), plan.empty_field()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for k in (1.0, 2.0, -1.0, 0.5):
        with torch.cuda.stream(a):
            work(beta, src, k, 20)
            done = a.record_event()
        b.wait_event(done)
        plan.stress(beta, out, stream=b)
        plan.flux(beta, 0.0, want_speed=False, stream=b, sigma=out, out=rhs)
        b.synchronize()
        want = plan.stress(src * k)
        assert torch.equal(out, want)
        assert torch.equal(rhs, plan.flux(src * k, 0.0, sigma=want)[0])
        a.wait_event(b.record_event())


def test_captured_kernels_after_an_event_see_the_other_branch():
    """A graph with two branches: one writes the field late, the other runs plan kernels before and after joining it."""
    shape = (32, 24, 32)
    plan = cdd.Plan([cdd.Instance(shape)], "f64")
    src = plan.pack([cdd.gaussian_random_field(shape, 0.06, 0.05, 4)])
    scale = torch.ones((), dtype=torch.float64, device="cuda")
    beta, out, first = torch.zeros_like(src), plan.empty_stress(), plan.empty_stress()
    big = torch.zeros(1 << 24, device="cuda")
    plan.stress(src, out)
    s, side = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        side.wait_event(s.record_event())
        with torch.cuda.stream(side):
            for _ in range(10):
                big.add_(1.0)
            torch.mul(src, scale, out=beta)
            done = side.record_event()
        plan.stress(src, first, stream=s)
        s.wait_event(done)
        plan.stress(beta, out, stream=s)
    for k in (1.0, -2.0, 3.0):
        scale.fill_(k)
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, plan.stress(src * k)) and torch.equal(first, plan.stress(src))


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_row_lines_that_leave_the_register_form(prec):
    """Line counts on a power-of-two axis that are no multiple of what the register-resident form needs run the two-pass
    form: the same bits in FP64, and in FP32 but for the order of the row sums (1e-6 rel-L2)."""
    shape = (12, 10, 64)
    b = np.random.default_rng(5).standard_normal((9,) + shape) * 0.05
    want = None
    for t in ({}, {"rows_lines": 8}, {"rows_lines": 1}, {"rows_lines": 7}):
        plan = cdd.Plan([cdd.Instance(shape)], prec, tuning=[t] if t else None)
        s = plan.stress(plan.pack([b]))
        want = s if want is None else want
        if prec == "f64":
            assert torch.equal(s, want), t
        else:
            assert float((s - want).norm()) < 1e-6 * float(want.norm()), t
