"""A species that is not finite makes temperature, tvirt and theta_v of its
point not finite in the same step, and the run stops (CFL violation) as soon in
mixed precision as in FP64, in the whole step and in the step split at the
physics."""
from __future__ import annotations

import numpy as np
import pytest

from regcm_gb300 import abi
from regcm_gb300 import case as cs
from regcm_gb300.moloch import CFLViolation, domain_from_case

pytestmark = pytest.mark.gpu

CROSS = ("t", "tvirt", "tetav", "rho", "qx", "ps")


def run(prec, value, species, where, split, boundary):
    """Non-finite masks of the cross-point fields after one step, and the step
    that stops the run."""
    case = cs.config1(50, 41, 12, precision=prec, apply_bdy=boundary)
    case.state["qx"][where][species] = value
    dom = domain_from_case(case)
    masks, stop = None, None
    for s in range(4):
        try:
            if split:
                dom.step_dynamics()
                dom.step_finish()
            else:
                dom.step(1)
        except CFLViolation:
            stop = s
        if s == 0:
            got = case.empty_state()
            dom.download(case.state_ptrs_of(got))
            masks = {n: ~np.isfinite(got[n]) for n in CROSS}
        if stop is not None:
            break
    dom.close()
    return masks, stop


# inside, in the relaxation zone and beside the ring; qv and a condensate
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("where,species", [((25, 20, 5), 0), ((4, 30, 8), 1), ((48, 39, 10), 0)])
@pytest.mark.parametrize("boundary", [True, False])
def test_mixed_follows_fp64(value, where, species, boundary):
    want, stop = run(abi.MLC_PREC_FP64, value, species, where, False, boundary)
    assert want["qx"].any() and want["tetav"].any()
    for split in (False, True):
        got, gstop = run(abi.MLC_PREC_MIXED, value, species, where, split, boundary)
        for n in CROSS:
            assert np.array_equal(got[n], want[n]), (split, n, got[n].sum(), want[n].sum())
        assert gstop == stop, split
