"""The kernels' scalar functions on arrays, each on the GPU against its plain
definition: reciprocal and quotient of few instructions (a rounding of the exact
value, inside their range and beyond its edges), -x/16 by the exponent, the WAF
limiter in both precisions, the threshold comparison and the saturation mixing
ratio."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from regcm_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = """
#include "mlc_scalar.cuh"
using namespace mlc;
template <class T, class F>
__global__ void each(const T *a, const T *b, T *out, int n, F f) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) out[e] = f(a[e], b[e]);
}
template <class T, class F>
int run(const T *a, const T *b, T *out, int n, F f) {
  T *d[3];
  for (T *&p : d)
    if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess) return 1;
  cudaMemcpy(d[0], a, n * sizeof(T), cudaMemcpyHostToDevice);
  cudaMemcpy(d[1], b, n * sizeof(T), cudaMemcpyHostToDevice);
  each<<<128, 128>>>(d[0], d[1], d[2], n, f);
  const cudaError_t e = cudaMemcpy(out, d[2], n * sizeof(T), cudaMemcpyDeviceToHost);
  for (T *p : d) cudaFree(p);
  return e != cudaSuccess;
}
extern "C" int f64(int what, const double *a, const double *b, double *out, int n) {
  switch (what) {
    case 0: return run(a, b, out, n, [] __device__(double x, double) { return recip_d(x); });
    case 1: return run(a, b, out, n, [] __device__(double x, double y) { return div_d(x, y); });
    case 2: return run(a, b, out, n, [] __device__(double x, double) { return neg_16th(x); });
    case 3: return run(a, b, out, n, [] __device__(double den, double num) {
      bool dbl;
      const double s = waf_sel(den, num, dbl);
      return twice(1.0, dbl) * s;
    });
    case 4: return run(a, b, out, n, [] __device__(double q, double c) { return below_pos<double>(q, c) ? 1.0 : 0.0; });
    case 5: return run(a, b, out, n, [] __device__(double t, double p) { return pfwsat_d(t, p); });
  }
  return 2;
}
extern "C" int f32(int what, const float *a, const float *b, float *out, int n) {
  if (what == 0) return run(a, b, out, n, [] __device__(float den, float num) { return waf_b(den, num); });
  return run(a, b, out, n, [] __device__(float x, float) { return neg_16th(x); });
}
"""
RECIP, DIV, NEG16, WAF, BELOW, PFWSAT = range(6)
INF, NAN, TINY = np.inf, np.nan, np.finfo(np.float64).smallest_subnormal


@pytest.fixture(scope="module")
def gpu(tmp_path_factory):
    d = tmp_path_factory.mktemp("scalar")
    (d / "scalar.cu").write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, "--extended-lambda", "-shared", "-I", str(build.CSRC),
                    "-o", str(d / "scalar.so"), str(d / "scalar.cu")], check=True, capture_output=True)
    lib = C.CDLL(str(d / "scalar.so"))

    def call(what, a, b=None):
        t = a.dtype
        a = np.ascontiguousarray(a)
        b = np.zeros_like(a) if b is None else np.ascontiguousarray(np.broadcast_to(b, a.shape).astype(t))
        out = np.empty_like(a)
        fn = lib.f64 if t == np.float64 else lib.f32
        p = lambda x: x.ctypes.data_as(C.c_void_p)
        assert fn(what, p(a), p(b), p(out), a.size) == 0
        return out

    return call


def around(x):
    x = np.asarray(x, dtype=np.float64)
    return np.concatenate([x, np.nextafter(x, INF), np.nextafter(x, -INF)])


def mantissas(rng, n):
    """Random mantissas in [1, 2), and those whose bits round in the extreme."""
    m = 1.0 + rng.random(n)
    edge = around([1.0, 1.5, 1.0 + 2.0**-23, 1.0 + 2.0**-24, 2.0 - 2.0**-23, 2.0 - 2.0**-24, 2.0 - 2.0**-52])
    return np.concatenate([m, edge[(edge >= 1.0) & (edge < 2.0)]])


def ulps(got, num, den):
    """|got - num/den| in units of got's last place, in extended precision."""
    g, a, b = (np.asarray(x, dtype=np.longdouble) for x in (got, num, den))
    return np.abs(g - a / b) / np.spacing(np.abs(got)).astype(np.longdouble)


SPECIAL = np.array([0.0, -0.0, INF, -INF, NAN, TINY, -TINY, 2.0**-1022, -(2.0**-1022), 1.7e308, -1.7e308, -1.0, -3.7])


def equal(a, b):
    return np.array_equal(a, b, equal_nan=True) and np.array_equal(np.signbit(a[a == 0]), np.signbit(b[b == 0]))


def test_reciprocal(gpu):
    """Inside FP32's range: e = 1 - x*r0 is below 1.5 * 2^-22 (the operand cut
    to 24 bits, two units of the FP32 reciprocal), so e^3 is below 2^-64, 2^-11
    units of the last place beside the final rounding's half."""
    rng = np.random.default_rng(1)
    x = np.concatenate([np.ldexp(mantissas(rng, 4000), e) for e in (-125, -124, -60, -7, -1, 0, 1, 9, 70, 124, 125)])
    assert ulps(gpu(RECIP, x), np.ones_like(x), x).max() <= 0.5 + 2.0**-10
    far = np.concatenate([around(np.ldexp(1.0, [-126, -125, 126, 127, -1000, 900])), SPECIAL])
    with np.errstate(all="ignore"):
        inside = (far >= 2.0**-125) & (far < 2.0**126)
        want = 1.0 / far
    got = gpu(RECIP, far)
    assert equal(got[~inside], want[~inside])
    assert ulps(got[inside], np.ones(inside.sum()), far[inside]).max() <= 0.5 + 2.0**-10


def test_quotient(gpu):
    """q = a*r is within two roundings of the quotient; corrected by the exact
    remainder, the error beside the final rounding's half is 2^-50 units."""
    rng = np.random.default_rng(2)
    a = rng.permutation(np.concatenate([np.ldexp(mantissas(rng, 4000), e) for e in (-766, -300, -1, 0, 3, 300, 767)]))
    a *= rng.choice([-1.0, 1.0], a.size)
    b = rng.permutation(np.concatenate([np.ldexp(mantissas(rng, 4000), e) for e in (-125, -60, -1, 0, 5, 60, 125)]))
    assert ulps(gpu(DIV, a, b), a, b).max() <= 0.5 + 2.0**-10
    exact = np.arange(1.0, 2000.0)
    assert np.array_equal(gpu(DIV, exact * 7.0, exact), np.full_like(exact, 7.0))
    x = np.concatenate([around(np.ldexp(1.0, [-768, -767, 769, 770])), SPECIAL])
    y = np.concatenate([around(np.ldexp(1.0, [-126, -125, 126])), SPECIAL, [3.0]])
    x, y = (v.ravel() for v in np.meshgrid(x, y))
    got = gpu(DIV, x, y)
    with np.errstate(all="ignore"):
        want = x / y
    finite = np.isfinite(want) & (want != 0)
    assert equal(got[~finite], want[~finite])
    assert np.abs(got[finite] / want[finite] - 1.0).max() <= 2.0**-52


def test_minus_a_sixteenth(gpu):
    rng = np.random.default_rng(3)
    x = np.concatenate([rng.standard_normal(4000) * 10.0 ** rng.uniform(-300, 300, 4000), SPECIAL,
                        around(np.ldexp(1.0, [-1022, -1019, -1018, -1017, 1023]))])
    assert equal(gpu(NEG16, x), -0.0625 * x)
    f = rng.standard_normal(4000).astype(np.float32)
    assert np.array_equal(gpu(1, f), np.float32(-0.0625) * f)


def limiter(den, num):
    """sign(den) * max(0, min(2d, max(q, min(2q, d)))), q = num*sign(den)"""
    t = den.dtype.type
    s = np.where(np.signbit(den), t(-1), t(1))
    q, d = num * s, np.abs(den)
    return s * np.maximum(t(0), np.minimum(d + d, np.maximum(q, np.minimum(q + q, d))))


def ratios(rng, scale, dtype):
    """den, num in every region of r = num/den and on its edges"""
    den = (scale * rng.standard_normal(6000)).astype(dtype)
    r = np.concatenate([rng.uniform(-3, 3, 5500), np.tile([-0.0, 0.0, 0.5, 1.0, 2.0], 100)]).astype(dtype)
    num = den * r
    num[5900:] = np.nextafter(num[5900:], np.where(np.arange(100) % 2, dtype(INF), dtype(-INF)))
    num[::89] = 0.0
    return den, num


@pytest.mark.parametrize("scale", [1e-20, 1e-3, 1.0, 300.0, 1e20])
def test_limiter_fp32(gpu, scale):
    den, num = ratios(np.random.default_rng(4), scale, np.float32)
    den[::97] = 0.0
    assert np.array_equal(gpu(0, den, num), limiter(den, num))


@pytest.mark.parametrize("scale", [1e-20, 1e-3, 1.0, 300.0, 1e20])
def test_limiter_fp64(gpu, scale):
    den, num = ratios(np.random.default_rng(5), scale, np.float64)
    assert np.array_equal(gpu(WAF, den, num), limiter(den, num))


def test_limiter_of_tiny_infinite_and_nan(gpu):
    """FP64 keeps the reference's guards of |den| < 1e-30: the limiter is 1 for
    |num| < 1e-30, else 0.  An infinite num is past every region; of a NaN the
    limiter stays finite in both precisions, between 0 and 2 den."""
    den = np.array([1e-31, -1e-31, 0.0, 1e-31, -9.9e-31])
    num = np.array([1e-32, 5.0, 0.0, -1e-31, -1e-29])
    assert np.array_equal(gpu(WAF, den, num), [1e-31, 0.0, 0.0, 1e-31, 0.0])
    den = np.array([2.0, -2.0, 2.0, -2.0])
    num = np.array([INF, INF, -INF, -INF])
    for t, what in ((np.float32, 0), (np.float64, WAF)):
        assert np.array_equal(gpu(what, den.astype(t), num.astype(t)), np.array([4.0, 0.0, 0.0, -4.0], t))
        b = gpu(what, den.astype(t), np.full(4, NAN, t))
        assert np.isfinite(b).all() and (b * den >= 0).all() and (np.abs(b) <= 4).all()


def test_threshold(gpu):
    rng = np.random.default_rng(6)
    for c in (1e-50, 1e-16, 1e-8, 0.01, 100.0, 1e10):
        q = np.concatenate([c * rng.uniform(-2, 2, 2000), around([c, 0.0, -c]), SPECIAL])
        assert np.array_equal(gpu(BELOW, q, c) != 0, q < c)


WATER = [0.209339997e-13, -0.373208410e-10, 0.892344772e-08, 0.196237241e-05, 0.305903558e-03, 0.264461437e-01,
         0.143064234e+01, 0.444007856e+02, 0.611213476e+03]
ICE = [0.262655803e-12, 0.149436277e-09, 0.387940929e-07, 0.602780717e-05, 0.614396778e-03, 0.420547422e-01,
       0.188369801e+01, 0.503109514e+02, 0.611123516e+03]


def test_saturation(gpu):
    """Against the polynomials in extended precision: nine roundings of partial
    sums no larger than the sum of the terms' magnitudes, then those of the cap,
    the difference, the quotient and the product, which p - es > 0.85 p keeps."""
    rng = np.random.default_rng(7)
    t = np.concatenate([273.15 + rng.uniform(-90, 120, 20000), 273.15 + around([-75.0, 0.0, 100.0])])
    p = np.exp(rng.uniform(np.log(50.0), np.log(1.1e5), t.size))
    td = np.clip(t - 273.15, -75.0, 100.0).astype(np.longdouble)
    es, size = np.zeros_like(td), np.zeros_like(td)
    for coef in (WATER, ICE):
        v, m = np.zeros_like(td), np.zeros_like(td)
        for c in coef:
            v, m = v * td + np.longdouble(c), m * np.abs(td) + abs(c)
        pick = (td >= 0) if coef is WATER else (td < 0)
        es, size = np.where(pick, v, es), np.where(pick, m, size)
    cap = np.longdouble(0.15) * p
    err = np.where(es < cap, size / es, 1.0) * 10 * 2.0**-53 + 6 * 2.0**-53
    es = np.minimum(es, cap)
    ep2 = np.longdouble(18.01528 / 28.96454)
    want = ep2 * es / (p - es)
    got = gpu(PFWSAT, t, p)
    assert (np.abs(got - want) / want <= 2.0 * err).all()
    assert np.isnan(gpu(PFWSAT, np.array([NAN, 280.0]), np.array([1e5, NAN]))).all()
