"""The forms of the column solve by segments and levels: a member gives the
same bits in batches whose size picks each form, with shallow and with deep
columns, and a deep domain that takes the streamed form agrees with the
oracle."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import Oracle
from regcm_gb300 import abi
from regcm_gb300 import case as cs
from regcm_gb300.moloch import MolochBatch, domain_from_case

from .conftest import rel_l2

pytestmark = pytest.mark.gpu

FP64, MIXED = abi.MLC_PREC_FP64, abi.MLC_PREC_MIXED


def dry(nx, ny, kz, prec=FP64):
    return cs.build(nx, ny, kz, dx=12000.0, dt=30.0, nsound=3, seed=nx + kz, wind=10.0,
                    hills=[(0.5 * nx * 12000.0, 0.5 * ny * 12000.0, 600.0)], theta_noise=0.3, tracer=True,
                    precision=prec, name=f"levels_{nx}x{ny}x{kz}")


# copies for six coefficient warps, three (none at these levels in the deep
# cases) and the streamed form: 192 segments a member, 56 in the deep ones
@pytest.mark.parametrize("prec,shape,copies", [(FP64, (70, 66, 9), (1, 3, 6)), (MIXED, (70, 66, 9), (1, 4, 13)),
                                               (FP64, (40, 30, 120), (1, 9)), (MIXED, (40, 30, 120), (1, 22))])
def test_forms_agree_bit_for_bit(prec, shape, copies):
    case, want = dry(*shape, prec=prec), None
    for n in copies:
        b = MolochBatch([case] * n)
        b.step(3)
        for m in {0, n - 1}:
            got = case.empty_state()
            b.download(m, case.state_ptrs_of(got))
            want = want or got
            for f in want:
                assert np.array_equal(want[f], got[f]), (n, m, f)
        b.close()


@pytest.mark.parametrize("nx,ny,kz", [(97, 140, 128), (130, 120, 101)])  # 3.6 and 3.9 segments an SM: streamed
def test_deep_domain_against_oracle(nx, ny, kz):
    """The one-step bound of the FP64 path, 1e-12 relative L2, in proportion to
    the levels above 41 (the rounding of Exner enters w over the layer depth)."""
    case = dry(nx, ny, kz)
    dom = domain_from_case(case)
    dom.step(1)
    got = case.empty_state()
    dom.download(case.state_ptrs_of(got))
    dom.close()
    orc = Oracle(case)
    st, _ = orc.step(1)
    assert st == 0
    ref = orc.state()
    orc.close()
    bad = {n: e for n in ("u", "v", "w", "pai", "tetav", "trac") if not (e := rel_l2(got[n], ref[n])) <= 1e-12 * kz / 41}
    assert not bad, bad
