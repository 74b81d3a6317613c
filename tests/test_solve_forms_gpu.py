"""The forms of the column solve (several warps a column, or a thread a column
with streamed planes, by the number of row segments): each against the oracle
at its edges - the fewest and most levels, row ends on and off a segment - and
bit for bit against the others, through the same member in batches of
different sizes."""
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


def dry(nx, ny, kz, prec=FP64, **kw):
    return cs.build(nx, ny, kz, dx=12000.0, dt=60.0, nsound=3, moist=False, seed=nx + kz, wind=10.0,
                    hills=[(0.5 * nx * 12000.0, 0.5 * ny * 12000.0, 600.0)], theta_noise=0.3, tracer=True,
                    precision=prec, name=f"dry_{nx}x{ny}x{kz}", **kw)


# 32-column segments a row times interior rows decides: at most 304 six
# coefficient warps, at most 1216 three, streamed above (FP64)
@pytest.mark.parametrize("nx,ny,kz", [(33, 30, 4), (32, 24, 5), (40, 26, 14), (64, 26, 128),     # six
                                      (97, 104, 5), (65, 160, 7),                               # three
                                      (191, 230, 4), (225, 190, 6)])                            # streamed
def test_fp64_step_against_oracle(nx, ny, kz):
    """The one-step bound of the FP64 path, 1e-12 relative L2 (the rounding of
    Exner enters w over the layer depth: in proportion above 41 levels)."""
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
    bound = 1e-12 * max(1.0, kz / 41.0)
    bad = {n: e for n in ("u", "v", "w", "pai", "tetav", "trac") if not (e := rel_l2(got[n], ref[n])) <= bound}
    assert not bad, bad


@pytest.mark.parametrize("prec,df", [(FP64, True), (MIXED, True), (MIXED, False)])
def test_forms_agree_bit_for_bit(prec, df):
    """A member alone (few segments: six warps) against itself in batches whose
    segments call for three warps and for the streamed form."""
    shape = (70, 66, 9)  # 192 segments
    case = dry(*shape, prec=prec)
    want = None
    for copies in (1, 4, 13):
        b = MolochBatch([dry(*shape, prec=prec) for _ in range(copies)])
        b.set_solve_precision(df)
        b.step(3)
        for m in {0, copies - 1}:
            got = case.empty_state()
            b.download(m, case.state_ptrs_of(got))
            if want is None:
                want = got
            for n in want:
                assert np.array_equal(want[n], got[n]), (copies, m, n)
        b.close()
