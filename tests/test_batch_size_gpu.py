"""A member's result does not depend on what else its context holds: the point
kernels run one level a thread in small contexts and four in large ones, and a
context whose thinnest frame is one point deep orders the step's end
differently.  Both precisions, bit for bit, over the step's forms and options:
rows and levels that fill no tile or chunk, TKE, nudging at the top, the
rotated pole's curvature, spectral nudging, the step split at the physics."""
from __future__ import annotations

import numpy as np
import pytest

from regcm_gb300 import abi
from regcm_gb300 import case as cs
from regcm_gb300.moloch import MolochBatch, domain_from_case

pytestmark = pytest.mark.gpu

PRECISIONS = [abi.MLC_PREC_FP64, abi.MLC_PREC_MIXED]


def build(nx, ny, kz, moist, prec, nadv=1, **kw):
    dx, dt, ns = (3000.0, 20.0, 4) if moist else (12000.0, 60.0, 3)
    return cs.build(nx, ny, kz, dx=dx, dt=dt, nsound=ns, nadv=nadv, moist=moist, seed=nx * ny, wind=12.0, jet=moist,
                    hills=[(0.4 * nx * dx, 0.6 * ny * dx, 700.0)], theta_noise=0.3, tracer=not moist,
                    precision=prec, name=f"batch_{nx}x{ny}x{kz}", **kw)


def member(b, m, case):
    got = case.empty_state()
    b.download(m, case.state_ptrs_of(got))
    return got


def same(a, b, where):
    for n in a:
        assert np.array_equal(a[n], b[n]), (where, n)


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("moist,kw", [(True, {"tke": True, "ipptls": 5}), (False, {"lrotllr": True, "nadv": 2}),
                                      (False, {"spectral": True, "dtrad": 60.0}), (True, {"apply_bdy": False})])
@pytest.mark.parametrize("prec", PRECISIONS)
def test_alone_and_in_a_large_batch(prec, moist, kw, split):
    case = build(69, 67, 10, moist, prec, **kw)  # 47 600 points: 54 copies are past the threshold (1.25 M)

    def run(copies):
        b = MolochBatch([case] * copies)
        for s in range(2):
            if split:
                b.step_dynamics()
                for m in range(copies):
                    t = case.tendencies(s)
                    b.set_tendencies(m, case.tend_ptrs_of(t))
                b.step_finish()
            else:
                b.step(1)
        got = [member(b, m, case) for m in (0, copies - 1)]
        b.close()
        return got

    want = run(1)[0]
    for m, got in enumerate(run(54)):
        same(want, got, m)


def ring_only(case):
    """The case without a relaxation zone: the boundary holds the ring alone."""
    for n in abi.IBND_FIELDS:
        case.static[n] = np.full_like(case.static[n], -1, order="F")
    return case


@pytest.mark.parametrize("moist", [False, True])
@pytest.mark.parametrize("prec", PRECISIONS)
def test_a_frame_one_point_deep(prec, moist):
    """A member whose frame is the ring: against the split step, which runs the
    passes one by one (FP64), and beside a member with a zone, whose result
    stays what it is alone."""
    plain, ring = build(41, 38, 7, moist, prec), ring_only(build(41, 38, 7, moist, prec))
    assert all((plain.static[n] > 0).any() for n in abi.IBND_FIELDS)
    b = MolochBatch([plain, ring])
    b.step(3)
    for m, case in enumerate((plain, ring)):
        dom = domain_from_case(case)
        dom.step(3)
        got = case.empty_state()
        dom.download(case.state_ptrs_of(got))
        dom.close()
        same(member(b, m, case), got, m)
    b.close()
    if prec == abi.MLC_PREC_FP64:
        whole, split = domain_from_case(ring), domain_from_case(ring)
        for _ in range(3):
            whole.step(1)
            split.step_dynamics()
            split.step_finish()
        a, c = ring.empty_state(), ring.empty_state()
        whole.download(ring.state_ptrs_of(a))
        split.download(ring.state_ptrs_of(c))
        whole.close()
        split.close()
        same(a, c, "split")
