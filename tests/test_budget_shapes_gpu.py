"""The allocation-free mass budget where its row split can go wrong: the
smallest extents, rows shorter and longer than a warp, one and several rows a
warp, and each species count its kernels are compiled for (2, 5, any)."""
from __future__ import annotations

import ctypes as C

import pytest

from regcm_gb300 import abi

from .test_zz_no_alloc import _fn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jx,iy,kz,nqx", [(5, 5, 1, 1), (6, 7, 2, 2), (34, 36, 3, 5), (35, 10, 5, 7), (36, 40, 4, 10),
                                          (97, 130, 41, 2), (260, 301, 60, 3), (70, 801, 40, 5)])
def test_budget_of_random_fields(jx, iy, kz, nqx):
    """Against FP64 sums of the same arrays: at most a few thousand roundings
    of the sum of magnitudes (2^-53 each), 1e-12 of it."""
    import torch
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(jx * 1000 + iy)
    f = lambda *s: torch.rand(*s, generator=gen, device=dev, dtype=torch.float64)
    rho, dz, qx = f(kz, iy - 1, jx - 1), f(kz, iy - 1, jx - 1), f(nqx, kz, iy - 1, jx - 1)
    u, v, ps = f(kz, iy - 1, jx) - 0.5, f(kz, iy, jx - 1) - 0.5, f(iy - 1, jx - 1)
    out = torch.full((7,), -1.0, dtype=torch.float64, device=dev)
    dims = abi.mlc_dims(jx, iy, kz, nqx, 0)
    dx, dt = 3000.0, 20.0
    rc = _fn()(C.byref(dims), dx, dt, *[a.data_ptr() for a in (rho, dz, qx, u, v, ps, out)],
               C.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
    assert rc == abi.MLC_OK
    m, q = rho * dz, qx.sum(0)
    fl = [u[..., 0] * m[..., 0], -u[..., -1] * m[..., -1], v[:, 0, 1:-1] * m[:, 0, 1:-1],
          -v[:, -1, 1:-1] * m[:, -1, 1:-1]]
    qf = [q[..., 0], q[..., -1], q[:, 0, 1:-1], q[:, -1, 1:-1]]
    inner = m[:, 1:-1, 1:-1]
    ref = [(dx * dx * inner, 1), (dt * dx, fl), (dx * dx * q[:, 1:-1, 1:-1] * inner, 1),
           (dt * dx, [a * b for a, b in zip(fl, qf)])]
    got = out.cpu().tolist()
    for n, (a, b) in enumerate(ref):
        terms = [a] if b == 1 else [a * t for t in b]
        want, size = sum(float(t.sum()) for t in terms), sum(float(t.abs().sum()) for t in terms)
        assert abs(got[n] - want) <= 1e-12 * size, n
    inner_ps = ps[1:-1, 1:-1]
    assert got[4] == float(inner_ps.max()) and got[5] == float(inner_ps.min()) and got[6] == 0.0
