"""The whole step's end (frame and interior point passes, winds, reduction)
where its split can go wrong: domains that are all frame, whose interior is a
few points, whose rows end on and off a 16-byte lane or a warp's columns; with
and without the boundary, tracers, TKE and the larger microphysics.  FP64
against the split step, which runs the passes one by one, bit for bit; mixed
members against themselves in a batch large enough for the longer level chunks."""
from __future__ import annotations

import numpy as np
import pytest

from regcm_gb300 import abi
from regcm_gb300 import case as cs
from regcm_gb300.moloch import MolochBatch, domain_from_case

pytestmark = pytest.mark.gpu


def build(nx, ny, kz, moist, prec=abi.MLC_PREC_FP64, **kw):
    dx, dt, ns = (3000.0, 20.0, 4) if moist else (12000.0, 60.0, 3)
    return cs.build(nx, ny, kz, dx=dx, dt=dt, nsound=ns, moist=moist, seed=nx * ny, wind=12.0, jet=moist,
                    hills=[(0.4 * nx * dx, 0.6 * ny * dx, 700.0)], theta_noise=0.3, tracer=not moist,
                    precision=prec, name=f"end_{nx}x{ny}x{kz}", **kw)


def state(dom, case):
    got = case.empty_state()
    dom.download(case.state_ptrs_of(got))
    return got


@pytest.mark.parametrize("nx,ny,kz,moist,kw", [
    (24, 21, 6, False, {}), (37, 36, 5, True, {}), (38, 41, 7, True, {"ipptls": 5}), (65, 23, 30, False, {"tke": True}),
    (130, 67, 23, False, {}), (67, 130, 9, True, {"lehmann": False}), (41, 39, 12, True, {"apply_bdy": False}),
    (129, 40, 8, True, {"ipptls": 1}), (64, 64, 41, True, {"tke": True})])
def test_whole_step_equals_split_step(nx, ny, kz, moist, kw):
    case = build(nx, ny, kz, moist, **kw)
    whole, split = domain_from_case(case), domain_from_case(case)
    for _ in range(3):
        dw = whole.step(1)
        split.step_dynamics()
        ds = split.step_finish()
        assert dw.ps_max == ds.ps_max and dw.ps_min == ds.ps_min
        assert dw.drymass == ds.drymass and dw.qadv == ds.qadv
    a, b = state(whole, case), state(split, case)
    whole.close()
    split.close()
    for n in a:
        assert np.array_equal(a[n], b[n]), n


@pytest.mark.parametrize("moist", [False, True])
def test_mixed_member_in_a_large_batch(moist):
    shape = (70, 66, 9)  # 62 of them pass the point kernels' one-level threshold
    case = build(*shape, moist, prec=abi.MLC_PREC_MIXED)
    dom = domain_from_case(case)
    dom.step(3)
    want = state(dom, case)
    dom.close()
    batch = MolochBatch([build(*shape, moist, prec=abi.MLC_PREC_MIXED) for _ in range(62)])
    batch.step(3)
    for m in (0, 61):
        got = case.empty_state()
        batch.download(m, case.state_ptrs_of(got))
        for n in want:
            assert np.array_equal(want[n], got[n]), (m, n)
    batch.close()
