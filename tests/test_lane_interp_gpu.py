"""The four-column interpolations between staggered and cross points of a
mixed member, where a row ends inside a lane or a tile: rows of one lane and a
remainder, just under and over 128 columns, and few levels.  Against the FP64
oracle after one step, within the mixed precision's one-step differences, and
a batch large enough for four levels a thread against the member alone."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import Oracle
from regcm_gb300 import abi
from regcm_gb300 import case as cs
from regcm_gb300.moloch import MolochBatch, domain_from_case

from .test_mixed_gpu import ONE_STEP_MAX

pytestmark = pytest.mark.gpu


def build(nx, ny, kz, prec, tke=False):
    return cs.build(nx, ny, kz, dx=3000.0, dt=20.0, nsound=4, moist=True, seed=nx, wind=12.0, jet=True,
                    hills=[(0.4 * nx * 3000.0, 0.6 * ny * 3000.0, 700.0)], theta_noise=0.3, tke=tke,
                    precision=prec, name=f"lane_{nx}x{ny}x{kz}")


def state_of(dom, case):
    got = case.empty_state()
    dom.download(case.state_ptrs_of(got))
    return got


@pytest.mark.parametrize("nx,ny,kz,tke", [(24, 25, 5, False), (34, 22, 7, True), (35, 30, 4, False),
                                          (127, 21, 6, False), (130, 23, 9, True), (133, 26, 6, False)])
def test_one_step_at_lane_edges(nx, ny, kz, tke):
    case = build(nx, ny, kz, abi.MLC_PREC_MIXED, tke)
    dom = domain_from_case(case)
    dom.step(1)
    got = state_of(dom, case)
    dom.close()
    orc = Oracle(build(nx, ny, kz, abi.MLC_PREC_FP64, tke))
    st, _ = orc.step(1)
    assert st == 0
    ref = orc.state()
    orc.close()
    for n, tol in ONE_STEP_MAX.items():
        assert np.abs(got[n] - ref[n]).max() <= tol * np.abs(ref[n]).max(), n


def test_four_levels_a_thread():
    shape = (131, 45, 11)  # 40 of them pass the one-level threshold
    cases = [build(*shape, abi.MLC_PREC_MIXED, True) for _ in range(40)]
    dom = domain_from_case(cases[0])
    dom.step(2)
    want = state_of(dom, cases[0])
    dom.close()
    batch = MolochBatch(cases)
    batch.step(2)
    got = cases[39].empty_state()
    batch.download(39, cases[39].state_ptrs_of(got))
    batch.close()
    for n in want:
        assert np.array_equal(got[n], want[n]), n
