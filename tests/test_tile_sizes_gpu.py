"""The horizontal WAF's tile width by size: rows of one, nearly one and just
over one tile of 32, 64 and 128 columns (the first and last tile write up to
the domain's edge), and rows past a block's last.  The tiles the rule picks
and every explicit shape give the same bits, in both precisions: the kernels'
roundings are explicit, so a member's result does not depend on the batch
that chose its tiles."""
from __future__ import annotations

import numpy as np
import pytest

from regcm_gb300 import abi
from regcm_gb300 import case as cs
from regcm_gb300.moloch import DEFAULT_SHAPES, domain_from_case

pytestmark = pytest.mark.gpu


def run(case, htile):
    dom = domain_from_case(case)
    if htile is not None:
        dom.set_launch_shapes(dict(DEFAULT_SHAPES, htile=htile))
    dom.step(2)
    got = case.empty_state()
    dom.download(case.state_ptrs_of(got))
    dom.close()
    return got


@pytest.mark.parametrize("prec", [abi.MLC_PREC_FP64, abi.MLC_PREC_MIXED])
@pytest.mark.parametrize("nx,ny,moist,kw", [
    (33, 22, True, {}), (34, 29, False, {}), (61, 26, False, {"lrotllr": True}), (65, 23, True, {}),
    (66, 31, False, {}), (125, 21, True, {"ipptls": 5}), (129, 27, True, {}), (130, 24, False, {}),
    (250, 22, False, {"lrotllr": True}), (253, 33, True, {"tke": True}), (254, 25, True, {})])
def test_tile_widths_same_bits(prec, nx, ny, moist, kw):
    dx, dt, ns = (3000.0, 20.0, 4) if moist else (12000.0, 60.0, 3)
    case = cs.build(nx, ny, 6, dx=dx, dt=dt, nsound=ns, moist=moist, seed=nx + ny, wind=12.0, jet=moist,
                    hills=[(0.4 * nx * dx, 0.6 * ny * dx, 700.0)], theta_noise=0.3, tracer=not moist,
                    precision=prec, name=f"tile_{nx}x{ny}", **kw)
    want = run(case, None)
    for htile in range(4):
        got = run(case, htile)
        for n in want:
            assert np.array_equal(got[n], want[n]), (htile, n)
