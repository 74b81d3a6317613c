"""Time-invariant fields derived on the device when a member is bound: rows
ending on and off a 32-byte sector, with and without a rotated pole and
relaxation zones.  In FP64 every product is a single rounding of the oracle's,
so one step is within the specified 1e-12; and a member that joins where a
larger one left (staging buffer and arena reused) equals the same member in a
fresh pool bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import Oracle
from regcm_gb300 import abi
from regcm_gb300 import case as cs
from regcm_gb300.moloch import MolochPool

from .test_parity_gpu import field_errors

pytestmark = pytest.mark.gpu


def build(nx, ny, kz, prec, **kw):
    return cs.build(nx, ny, kz, dx=12000.0, dt=60.0, nsound=3, moist=False, seed=nx, wind=12.0,
                    hills=[(0.4 * nx * 12000.0, 0.6 * ny * 12000.0, 700.0)], theta_noise=0.3, tracer=True,
                    precision=prec, name=f"bind_{nx}x{ny}x{kz}", **kw)


def run(pool, case):
    slot = pool.join(case)
    pool.step(1)
    got = case.empty_state()
    pool.download(slot, case.state_ptrs_of(got))
    pool.leave(slot)
    return got


@pytest.mark.parametrize("kw", [{}, {"lrotllr": True}, {"apply_bdy": False}])
@pytest.mark.parametrize("prec", [abi.MLC_PREC_FP64, abi.MLC_PREC_MIXED])
def test_bound_after_another(prec, kw):
    cases = [build(nx, ny, kz, prec, **kw) for nx, ny, kz in ((61, 43, 12), (33, 36, 7), (40, 29, 12), (34, 51, 5))]
    pool = MolochPool(cases[0].params, 2)
    for case in cases:
        got = run(pool, case)
        fresh = MolochPool(case.params, 1)
        want = run(fresh, case)
        fresh.close()
        for n in want:
            assert np.array_equal(got[n], want[n]), (case.name, n)
        if prec == abi.MLC_PREC_FP64:
            orc = Oracle(case)
            st, _ = orc.step(1)
            assert st == 0
            errs = field_errors(got, orc.state(), case)
            orc.close()
            assert max(errs.values()) <= 1e-12, (case.name, errs)
    pool.close()
