"""Stencil planes staged with wrapped asynchronous copies (edge tiles, narrow grids, rows of 4 k + 2 values,
fields that are not 16-byte aligned) and every split of the march along axis 0, against the CPU oracle.

Tolerances as for the staged planes of the wider grids: FP64 1e-12, FP32 5e-6 rel-L2.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import cdd
import cdd_oracle as O

TOL = {"f64": 1e-12, "f32": 5e-6}
LOAD = (-0.025, -0.025, 0.05)


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


def setup(shape, prec, planes=0, shift=0):
    b = cdd.gaussian_random_field(shape, 0.08, 0.05, 11)
    if prec == "f32":
        b = b.astype(np.float32).astype(np.float64)
    plan = cdd.Plan([cdd.Instance(shape, load_rate=LOAD)], prec,
                    tuning=[{"stencil_planes": planes}] if planes else None)
    beta = plan.pack([b])
    if shift:   # the same field `shift` elements past a 256-byte boundary
        wide = torch.zeros(plan.field_elems + shift, dtype=plan.dtype, device=plan.device)
        wide[shift:] = beta
        beta = wide[shift:]
    return b, plan, beta


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(4, 4, 4), (6, 8, 18), (8, 10, 32), (4, 6, 20), (6, 4, 36), (8, 12, 40),
                                   (4, 18, 54), (4, 9 * 2, 64), (6, 20, 100), (4, 4), (18, 6), (10, 36), (20, 162)])
def test_flux_of_every_staging_against_oracle(shape, prec):
    b, plan, beta = setup(shape, prec)
    rhs, speed = plan.flux(beta, 0.1)
    ref, ref_speed = O.full_flux(b, 0.1, O.Params(load_rate=np.array(LOAD)))
    assert rel(plan.field_view(rhs, 0).cpu().numpy(), ref) < TOL[prec]
    assert rel(speed.cpu().numpy().reshape(shape), ref_speed) < TOL[prec]
    plan.check_status()


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(12, 20, 72), (10, 24, 54), (9 * 2, 16, 32)])
def test_planes_per_block_and_field_alignment_change_no_bit(shape, prec):
    _, plan, beta = setup(shape, prec)
    sigma = plan.stress(beta)
    want, want_speed = plan.flux(beta, 0.1, sigma=sigma)
    for planes, shift in [(1, 0), (2, 0), (5, 0), (64, 0), (0, 1), (0, 2), (3, 1)]:
        _, other, field = setup(shape, prec, planes, shift)
        rhs, speed = other.flux(field, 0.1, sigma=sigma)
        assert torch.equal(rhs, want) and torch.equal(speed, want_speed)
        other.check_status()
