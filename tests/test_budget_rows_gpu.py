"""The allocation-free mass budget of domains with few, long rows, whose rows
are split over warps: against FP64 sums of the same arrays, as
tests/test_budget_shapes_gpu.py."""
from __future__ import annotations

import pytest

from .test_budget_shapes_gpu import test_budget_of_random_fields as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jx,iy,kz,nqx", [(30001, 5, 1, 5), (1025, 9, 4, 2), (98, 7, 3, 3), (99, 5, 1, 5), (131, 33, 20, 5),
                                          (67, 44, 41, 5), (2001, 122, 31, 1)])
def test_budget_of_long_rows(jx, iy, kz, nqx):
    check(jx, iy, kz, nqx)
