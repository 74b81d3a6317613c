"""The end of steps that nudge spectrally, four columns a lane in mixed members:
bit for bit the split step's, which runs the same expressions a point a thread,
where rows end on and off a lane or a tile, with and without tracers and the
larger microphysics, and over the species' floors."""
from __future__ import annotations

import numpy as np
import pytest

from regcm_gb300 import abi
from regcm_gb300 import case as cs
from regcm_gb300.moloch import domain_from_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [abi.MLC_PREC_FP64, abi.MLC_PREC_MIXED])
@pytest.mark.parametrize("nx,ny,kz,kw", [(64, 33, 9, {"moist": True}), (65, 34, 10, {"tracer": True}),
                                         (66, 41, 7, {"moist": True, "ipptls": 5}), (131, 40, 4, {"moist": True, "ipptls": 1}),
                                         (128, 45, 12, {"moist": True, "tke": True, "ipptls": 4})])
def test_whole_step_equals_split_step(nx, ny, kz, kw, prec):
    moist = kw.get("moist", False)
    case = cs.build(nx, ny, kz, dx=12000.0, dt=60.0, nsound=3, seed=nx + ny, wind=12.0, jet=moist, theta_noise=0.3,
                    hills=[(0.4 * nx * 12000.0, 0.6 * ny * 12000.0, 700.0)], spectral=True, dtrad=120.0,
                    precision=prec, name=f"spec_{nx}x{ny}x{kz}", **kw)
    case.state["qx"][::5, ::3, ::2, 1] = -1e-6  # below its floor
    if "trac" in case.state:
        case.state["trac"][::4, ::5, ::3] = -1e-3
    whole, split = domain_from_case(case), domain_from_case(case)
    for _ in range(3):
        whole.step(1)
        split.step_dynamics()
        split.step_finish()
    a, b = case.empty_state(), case.empty_state()
    whole.download(case.state_ptrs_of(a))
    split.download(case.state_ptrs_of(b))
    whole.close()
    split.close()
    for n in a:
        assert np.array_equal(a[n], b[n]), n
