// mlc_advect.cu -- WAF flux-form advection of every advected field
// (Main/mod_moloch.F90:767-1042, subroutines advection and wafone, with the
// interpolations of :1445-1569 and local_flow_param :1571-1590).
//
//   adv_prep        u,v -> ux,vx (4th order, 2nd at the edges) and w -> wx.
//   adv_vertical    a thread a column and field (FP32 in large launches two
//                   fields): both vertical WAF passes (do_vadvtwice), streamed
//                   upward through registers.
//   adv_horizontal  per tile (a warp a row, 32 to 128 columns) and level, field
//                   by field: meridional then zonal WAF.  The tile's wz lands in
//                   shared memory with a 2-point halo; from it come the
//                   meridional fluxes and the intermediate p0 on a 2-column
//                   halo, then the zonal fluxes and the result, so each field
//                   is read and written once.  The result goes to a second
//                   buffer because the halo columns of a tile still need the
//                   field's old values.
//   adv_curvature   curvature terms on ux, vx (skipped when they are zero at
//                   every point: with uniform map factors the reference adds
//                   an exact zero).
//   adv_back        ux,vx -> u,v and wx -> w (4th order, 2nd at the edges).
// The fluxes are formed per unit wind and the wind joins the cells' metric
// factors, and an update's terms are summed before the field (waf_g, waf_update,
// vupdate): the reference's sums with other operand orders, equal to rounding.
// The interpolations and curvature terms follow the reference's expressions.
// The ratios dtrdz*fmz/fmzf of the vertical passes are per-domain constants read
// from arrays computed once with the same expression.
#include <type_traits>

#include "mlc_kernels.cuh"
#include "mlc_scalar.cuh"
#include "mlc_tma.cuh"

namespace mlc {

namespace {

// x + (gs*cs - gn*cn + dv*p): a WAF update from the fluxes per unit wind of a
// cell's two faces, the faces' winds times the cell's metric factors, the
// divergence factor and the field before the update.  The terms, which nearly
// cancel, are summed before x.  Every rounding is explicit, so the tile shapes
// give the same bits.
template <class T>
__device__ __forceinline__ T waf_update(T x, T gs, T cs, T gn, T cn, T dv, T p) {
  return x + fma_r(gs, cs, fma_r(-gn, cn, mul_r(dv, p)));
}

// The upwind tests zamu >= 0 and zamu > 0.  For FP64 they are made on the
// bit pattern by the integer pipe (each FP64 compare is an instruction of the
// 1/64-rate FP64 pipe on GB300), with the comparisons' exact results for
// -0, infinities and NaN; FP32 compares directly.
template <class T>
__device__ __forceinline__ bool nonneg(T x) {
  if constexpr (sizeof(T) == sizeof(double)) {
    const long long b = bits_of(x);
    return (b >= 0 && b <= 0x7ff0000000000000LL) || b == (long long)0x8000000000000000ULL;
  } else {
    return x >= T(0);
  }
}
template <class T>
__device__ __forceinline__ bool positive(T x) {
  if constexpr (sizeof(T) == sizeof(double)) {
    const long long b = bits_of(x);
    return b > 0 && b <= 0x7ff0000000000000LL;
  } else {
    return x > T(0);
  }
}

// a - a for the limiter's region tests: +0 for a finite a, else a NaN (every
// NaN takes the same region), formed on the integer pipe in FP64
template <class T>
__device__ __forceinline__ T self_diff(T a) {
  if constexpr (sizeof(T) == sizeof(double)) {
    const long long b = bits_of(a);
    const long long e = 0x7ff0000000000000LL;
    return (b & e) == e ? __longlong_as_double(0x7ff8000000000000LL) : 0.0;
  } else {
    return a - a;
  }
}
// The WAF flux (mlc_scalar.cuh) per unit wind: vel*g with vel = 2*hvel (the wind itself),
// g = x - zmih*B, x = a upwind of a positive zamu (is = +1) else c, and
// zmih = (zamu - is)/2: (a + c) - is*den = 2x exactly, so in exact arithmetic
//   hvel*((a + c) - (is*den + (zamu - is)*B)) = vel*(x - zmih*B).
// One fused multiply-add; the wind joins the cells' metric factors, formed
// once for every field (FP64, moist 512x512x41, a step: horizontal WAF 4.90 ms
// with the wind in every flux, 3.65 so; vertical 2.35 and 1.82).
// g with den = c - a and the upwind value x given (an interface's den is the
// num of the interfaces on either side: a caller that has the neighbouring
// differences forms each once); nz = -zmih
template <class T>
__device__ __forceinline__ T waf_g(T nz, T x, T den, T num) {
  if constexpr (sizeof(T) == sizeof(double)) {
    bool dbl;
    const double sel = waf_sel(den, num, dbl);
    return __fma_rn(twice(nz, dbl), sel, x);
  } else {
    return fmaf(nz, waf_b(den, num), x);
  }
}
// -zmih = (is - zamu)/2 of an interface
template <class T>
__device__ __forceinline__ T waf_nz(T zamu, bool up) {
  return fma_r(T(-0.5), zamu, up ? T(0.5) : T(-0.5));
}

// The advected fields of a member, in the reference's order (tetav, pai,
// ux, vx, wx, qv, qx(iqfrst:nqx) when ipptls > 0, tkex when ibltyp = 2,
// trac; advection, Main/mod_moloch.F90:781-807).  Table 0 holds the fields of type R: all of
// them in FP64, all but theta_v and Exner in a mixed member, whose two FP64
// fields form table 1.  cur is the field's current half, out the other.
template <class R>
__device__ __forceinline__ int n_table_r(const Dom<R> &D) {
  const int nfix = sizeof(R) == sizeof(double) ? 2 : 0;
  return nfix + 4 + (D.c.ipptls > 0 ? D.g.nqx - 1 : 0) + D.c.tke + D.g.ntr;
}

template <class R>
__device__ __forceinline__ void field_r(const Dom<R> &D, int f, int adv, const R *&cur, R *&out) {
  if (sizeof(R) == sizeof(double)) {
    if (f == 0) { cur = (const R *)D.tetav[adv]; out = (R *)D.tetav[adv ^ 1]; return; }
    if (f == 1) { cur = (const R *)D.pai[adv]; out = (R *)D.pai[adv ^ 1]; return; }
    f -= 2;
  }
  const size_t F = D.g.field3();
  switch (f) {
    case 0: cur = D.ux[adv]; out = D.ux[adv ^ 1]; return;
    case 1: cur = D.vx[adv]; out = D.vx[adv ^ 1]; return;
    case 2: cur = D.wx[adv]; out = D.wx[adv ^ 1]; return;
    case 3: cur = D.qx[adv]; out = D.qx[adv ^ 1]; return;
    default: break;
  }
  f -= 4;
  const int nq = D.c.ipptls > 0 ? D.g.nqx - 1 : 0;
  if (f < nq) {
    cur = D.qx[adv] + (size_t)(f + 1) * F;
    out = D.qx[adv ^ 1] + (size_t)(f + 1) * F;
    return;
  }
  f -= nq;
  if (D.c.tke) {
    if (f == 0) {
      cur = D.tkex[adv];
      out = D.tkex[adv ^ 1];
      return;
    }
    f -= 1;
  }
  cur = D.trac[adv] + (size_t)f * F;
  out = D.trac[adv ^ 1] + (size_t)f * F;
}

// The field set `set` of a member: 0 = the R table, 1 = the FP64 table.
template <class R, class T>
__device__ __forceinline__ void field_t(const Dom<R> &D, int set, int f, int adv, const T *&cur,
                                        T *&out, T *&wz) {
  if constexpr (sizeof(T) == sizeof(R)) {
    const R *c0;
    R *o0;
    field_r<R>(D, f, adv, c0, o0);
    cur = (const T *)c0;
    out = (T *)o0;
    wz = (T *)D.wz[f];
  } else {
    (void)set;
    cur = f == 0 ? D.tetav[adv] : D.pai[adv];
    out = f == 0 ? D.tetav[adv ^ 1] : D.pai[adv ^ 1];
    wz = D.wz_d[f];
  }
}

template <class R, int LV>
__global__ void k_adv_prep(const Dom<R> *__restrict__ doms, int uvoff, int advoff, int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const int uv = (D.clk->uv_role + uvoff) & 1, adv = (D.clk->adv_role + advoff) & 1;
  const R *__restrict__ u = D.u[uv];
  const R *__restrict__ v = D.v[uv];
  const R *__restrict__ w = D.w;
  R *__restrict__ ux = D.ux[adv];
  R *__restrict__ vx = D.vx[adv];
  R *__restrict__ wx = D.wx[adv];
  const Pt q_ = point_at<LV>(wi, 1, 1);
  const int j = q_.j, k0 = q_.k;
  if (k0 > g.kz) return;
  const int i = q_.i;
  const int jx = g.jx, iy = g.iy, kz = g.kz;
  if (j > jx - 1 || i > iy - 1) return;
  const size_t ij = g.at2(j, i), PS = g.PS, S = (size_t)g.P;
#pragma unroll
  for (int k = k0; k < k0 + LV && k <= g.kz; ++k) {
    const size_t o = ij + (size_t)(k - 1) * PS;
    // uvstagtouvx :1535-1549
    R a;
    if (j == 1) a = R(0.5) * (u[o] + u[o + 1]);
    else if (j == jx - 1) a = R(0.5) * (u[o + 1] + u[o]);
    else a = interp4<R>(u[o + 1], u[o], u[o + 2], u[o - 1]);
    ux[o] = a;
    // :1553-1566
    if (i == 1) a = R(0.5) * (v[o] + v[o + S]);
    else if (i == iy - 1) a = R(0.5) * (v[o + S] + v[o]);
    else a = interp4<R>(v[o + S], v[o], v[o + 2 * S], v[o - S]);
    vx[o] = a;
    // zstagtoh :1445-1459
    if (k == 1) a = R(0.5) * (w[o + PS] + w[o]);
    else if (k == kz) a = R(0.5) * (w[o + PS] + w[o]);
    else a = interp4<R>(w[o + PS], w[o], w[o + 2 * PS], w[o - PS]);
    wx[o] = a;
    if (D.c.tke) {
      // zstagtoh(tke, tkex) (Main/mod_moloch.F90:782-784)
      const R *__restrict__ tk = D.tke;
      if (k == 1 || k == kz) a = R(0.5) * (tk[o + PS] + tk[o]);
      else a = interp4<R>(tk[o + PS], tk[o], tk[o + 2 * PS], tk[o - PS]);
      D.tkex[adv][o] = a;
    }
    if constexpr (sizeof(R) == sizeof(double)) {
      // the vertical WAF's factors, once for all fields (FP64 arithmetic is
      // the FP64 path's bound): s(k)*zu(k) and s(k+1)*zd(k) of the level's
      // fluxes, their difference, and -zmih of interface k+1, whose sign bit
      // of zamu's factor s(k+1) says which side is upwind
      const double skp = D.s[o + PS];
      const double cu = __dmul_rn(D.s[o], D.sa.zrfmu[o]), cd = __dmul_rn(skp, D.sa.zrfmd[o]);
      D.vcu[o] = cu;
      D.vcd[o] = cd;
      D.vdiv[o] = cu - cd;
      const double zamu = __dmul_rn(skp, 0.5 * (D.c.dtstepa * D.c.rdzita));
      D.vnz[o] = waf_nz<double>(zamu, nonneg(zamu));
    }
  }
}

// ---- lane vectors ---------------------------------------------------------
template <int B> struct VecOf;
template <> struct VecOf<4> { using t = unsigned; };
template <> struct VecOf<8> { using t = uint2; };
template <> struct VecOf<16> { using t = uint4; };

// v consecutive elements at p, which is aligned to min(v * sizeof(T), 16)
template <class T, int V>
__device__ __forceinline__ void ld_vec(T (&x)[V], const T *p) {
  constexpr int B = V * (int)sizeof(T);
  if constexpr (B <= 16) {
    const typename VecOf<B>::t w = *reinterpret_cast<const typename VecOf<B>::t *>(p);
    memcpy(x, &w, B);
  } else {
#pragma unroll
    for (int h = 0; h < B / 16; ++h) {
      const uint4 w = reinterpret_cast<const uint4 *>(p)[h];
      memcpy(reinterpret_cast<char *>(x) + 16 * h, &w, 16);
    }
  }
}
template <class T, int V>
__device__ __forceinline__ void st_vec(T *p, const T (&x)[V]) {
  constexpr int B = V * (int)sizeof(T);
  if constexpr (B <= 16) {
    typename VecOf<B>::t w;
    memcpy(&w, x, B);
    *reinterpret_cast<typename VecOf<B>::t *>(p) = w;
  } else {
#pragma unroll
    for (int h = 0; h < B / 16; ++h) {
      uint4 w;
      memcpy(&w, reinterpret_cast<const char *>(x) + 16 * h, 16);
      reinterpret_cast<uint4 *>(p)[h] = w;
    }
  }
}
// the lane's v elements of row r (1-based) of a plane, or zeros
template <class T, int V>
__device__ __forceinline__ void ld_row(T (&x)[V], const T *plane, int e0, int r, unsigned P, bool ok) {
  if (ok) {
    ld_vec<T, V>(x, plane + (unsigned)e0 + (unsigned)(r - 1) * P);
  } else {
#pragma unroll
    for (int q = 0; q < V; ++q) x[q] = T(0);
  }
}
// element q+1 of the lane's columns: the lane's own, or the next lane's first
template <class T, int V>
__device__ __forceinline__ void next_col(T (&e)[V], const T (&x)[V]) {
#pragma unroll
  for (int q = 0; q + 1 < V; ++q) e[q] = x[q + 1];
  e[V - 1] = __shfl_down_sync(0xffffffffu, x[0], 1);
}

// Four FP32 points of a row interpolated from the eight around them
__device__ __forceinline__ void interp_vec(float (&x)[4], const float (&a)[4], const float (&b)[4], const float (&c)[4],
                                           const float (&d)[4], bool edge) {
#pragma unroll
  for (int q = 0; q < 4; ++q) x[q] = edge ? interp2<float>(a[q], b[q]) : interp4<float>(a[q], b[q], c[q], d[q]);
}
// x stored at p where e0 + q < n (0-based columns)
__device__ __forceinline__ void store_row4(float *p, const float (&x)[4], int e0, int n) {
  if (e0 + 4 <= n) {
    st_vec<float, 4>(p, x);
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (e0 + q < n) p[q] = x[q];
  }
}

// k_adv_prep of a mixed member in lanes of four columns: 16-byte loads of the
// rows and levels around a point, w's carried from level to level, so a point
// takes three loads instead of twelve (moist 512x512x41: 57 us a step
// against 92).  Block 32 lanes x 4 rows, grid as k_sound_div_v4's.
template <class R, int LV>
__global__ void __launch_bounds__(128) k_adv_prep_v4(const Dom<R> *__restrict__ doms, int uvoff, int advoff,
                                                     int tiles_j, const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const int jx = g.jx, iy = g.iy, kz = g.kz;
  const int e0 = ((int)wi.a * 32 + (int)threadIdx.x) * 4, i = (int)wi.b * 4 + (int)threadIdx.y + 1;
  const int k0 = (int)wi.c * LV + 1;
  if (e0 + 1 > jx - 1 || i > iy - 1 || k0 > kz) return;
  const int uv = (D.clk->uv_role + uvoff) & 1, adv = (D.clk->adv_role + advoff) & 1;
  const unsigned P = (unsigned)g.P, PS = (unsigned)g.PS, ij = (unsigned)e0 + (unsigned)(i - 1) * P;
  const float *__restrict__ u = D.u[uv] + ij;
  const float *__restrict__ v = D.v[uv] + ij;
  const float *__restrict__ w = D.w + ij;
  const float *__restrict__ tk = D.c.tke ? D.tke + ij : nullptr;
  float *__restrict__ ux = D.ux[adv] + ij;
  float *__restrict__ vx = D.vx[adv] + ij;
  float *__restrict__ wx = D.wx[adv] + ij;
  float *__restrict__ tkx = D.c.tke ? D.tkex[adv] + ij : nullptr;
  float w0[4] = {}, w1[4], w2[4], w3[4] = {};  // w at levels k-1 .. k+2
  unsigned o = (unsigned)(k0 - 1) * PS;
  if (k0 >= 2) ld_vec<float, 4>(w0, w + o - PS);
  ld_vec<float, 4>(w1, w + o);
  ld_vec<float, 4>(w2, w + o + PS);
  for (int k = k0; k < k0 + LV && k <= kz; ++k, o += PS) {
    float x[4];
    {
      // uvstagtouvx :1535-1549: columns e0-1 .. e0+5
      float a[7] = {};
      float m[4];
      ld_vec<float, 4>(m, u + o);
      if (e0 >= 1) a[0] = (u + o)[-1];  // (o may be 0: no unsigned o - 1)
#pragma unroll
      for (int q = 0; q < 4; ++q) a[1 + q] = m[q];
      if (e0 + 4 <= jx - 1) a[5] = u[o + 4];
      if (e0 + 5 <= jx - 1) a[6] = u[o + 5];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int j = e0 + q + 1;
        x[q] = j == 1 || j == jx - 1 ? interp2<float>(a[q + 1], a[q + 2])
                                     : interp4<float>(a[q + 2], a[q + 1], a[q + 3], a[q]);
      }
      store_row4(ux + o, x, e0, jx - 1);
    }
    {
      // :1553-1566: rows i-1 .. i+2
      float a[4] = {}, b[4], c[4], d[4] = {};
      if (i >= 2) ld_vec<float, 4>(a, v + o - P);
      ld_vec<float, 4>(b, v + o);
      ld_vec<float, 4>(c, v + o + P);
      if (i <= iy - 2) ld_vec<float, 4>(d, v + o + 2 * P);
      interp_vec(x, c, b, d, a, i == 1 || i == iy - 1);
      store_row4(vx + o, x, e0, jx - 1);
    }
    // zstagtoh :1445-1459
    if (k < kz) ld_vec<float, 4>(w3, w + o + 2 * PS);
    interp_vec(x, w2, w1, w3, w0, k == 1 || k == kz);
    store_row4(wx + o, x, e0, jx - 1);
    if (tk) {
      // zstagtoh(tke, tkex) (Main/mod_moloch.F90:782-784)
      float a[4] = {}, b[4], c[4], d[4] = {};
      if (k >= 2) ld_vec<float, 4>(a, tk + o - PS);
      ld_vec<float, 4>(b, tk + o);
      ld_vec<float, 4>(c, tk + o + PS);
      if (k < kz) ld_vec<float, 4>(d, tk + o + 2 * PS);
      interp_vec(x, c, b, d, a, k == 1 || k == kz);
      store_row4(tkx + o, x, e0, jx - 1);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) { w0[q] = w1[q]; w1[q] = w2[q]; w2[q] = w3[q]; }
  }
}

// Two vertical WAF passes (do_vadvtwice, :858-922), one thread per column
// and field, streaming the levels upward through registers.  Pass 1's flux
// at interface k+1 needs the input at levels k-1..k+2 and its update at k the
// fluxes at k and k+1; pass 2 needs pass 1's output at m-1..m+2, so it runs
// two levels behind pass 1 in the same loop.  Every value is loaded once and
// the column never touches shared memory.  R is the type of the winds and
// metric, T that of the advected field and of the arithmetic.
// the flux per unit s through interface k+1 between levels k and k+1, its
// upwind difference col(k1) - col(k1p1) with the reference's clamps
// k1p1 = min(k+2, kz), k1 = max(k-1, 1); d: the differences c(k) - c(k+1) of
// the interface itself, of the one above it (k-1, k) and below it (k+1, k+2)
template <class T>
__device__ __forceinline__ T vflux(T nz, bool up, T ck, T cp1, T d_above, T d, T d_below, int k, int kz) {
  const T num = up ? (k + 2 <= kz ? d_below : self_diff<T>(cp1)) : (k >= 2 ? d_above : self_diff<T>(ck));
  return waf_g<T>(nz, up ? cp1 : ck, d, num);
}
// (levels inside, where no clamp acts)
template <class T>
__device__ __forceinline__ T vflux_in(T nz, bool up, T ck, T cp1, T d_above, T d, T d_below) {
  return waf_g<T>(nz, up ? cp1 : ck, d, up ? d_below : d_above);
}
// pk - gb*cu + ga*cd + dv*pk: gb, ga the fluxes per unit s of the interfaces
// above and below, cu and cd s times their metric ratios, dv = cu - cd
template <class T>
__device__ __forceinline__ T vupdate(T pk, T gb, T ga, T dv, T cu, T cd) {
  return fma_r(dv, pk, fma_r(ga, cd, fma_r(-gb, cu, pk)));
}

// Blocks of 256 threads an SM the vertical WAF is compiled for, FP64 and FP32
// (0: no bound, the compiler's own register choice).  Moist 512x512x41 step:
// FP32, one field a thread, 3/4/5/6 blocks 309/283/252/313 us; two fields
// 3/4/5 blocks 220/212/318; FP64 2 (by its registers) and 3 1820 and 1988.
#ifndef MLC_VERT_MINB_D
#define MLC_VERT_MINB_D 0
#endif
#ifndef MLC_VERT_MINB_F
#define MLC_VERT_MINB_F 5
#endif
#ifndef MLC_VERT_MINB_2
#define MLC_VERT_MINB_2 4
#endif
template <class T, int NF>
constexpr int vert_min_blocks() {
  if (sizeof(T) == sizeof(double)) return MLC_VERT_MINB_D > 0 ? MLC_VERT_MINB_D : 1;
  return NF == 2 ? MLC_VERT_MINB_2 : MLC_VERT_MINB_F;
}
// a pointer into a field as one to global memory (fields are picked from a
// table, which hides that from the compiler)
template <class T>
__device__ __forceinline__ T *global_ptr(T *p) {
  return (T *)__cvta_global_to_generic(__cvta_generic_to_global((const void *)p));
}
// Fields f0 .. f0+NF-1 of the column (j, i), both passes.  FP32 members of
// large launches take two fields a thread, which share the level's loads and
// factors: the kernel is bound by instructions (54 against 119 a level and
// field; moist 512x512x41 0.256 -> 0.212 ms a step, 32 members of 128x128x30
// 0.239 -> 0.207).  Small ones need the threads (64x64x30 15.0 us against
// 14.2).  Copies further ahead (a shared-memory ring of 3 to 8 levels) gained
// nothing.
template <class R, class T, int NF>
__device__ __forceinline__ void vertical_column(const Dom<R> &D, int set, int f0, int adv, size_t ij) {
  const Scal &c = D.c;
  const int kz = D.g.kz;
  const T *src[NF];
  T *dst[NF];
#pragma unroll
  for (int n = 0; n < NF; ++n) {
    T *outp;
    field_t<R, T>(D, set, f0 + n, adv, src[n], outp, dst[n]);
    (void)outp;
    src[n] = global_ptr(src[n]) + ij;
    dst[n] = global_ptr(dst[n]) + ij;
  }
  const R *__restrict__ sp = D.s + ij;
  const R *__restrict__ zup = D.sa.zrfmu + ij;
  const R *__restrict__ zdp = D.sa.zrfmd + ij;
  const unsigned PS = (unsigned)D.g.PS;  // a domain's fields stay below 2^31 elements
  // -1/2 of the factor of s in zamu
  const T hdtrdz = T(-0.25) * (pick<T>(c.dtstepa, c.dtstepaf) * pick<T>(c.rdzita, c.rdzitaf));

  // windows: pass-1 input at k..k+1, pass-1 output at k-2..k-1, levels k-2 and
  // k-1 as loaded, the pass-1 flux at interface k and the pass-2 flux at
  // interface k-2, and the differences c(k) - c(k+1) of the pass-1 input at
  // interfaces k-1, k and of the pass-2 input at m-1, m (m = k-2)
  constexpr bool kPre = sizeof(R) == sizeof(double) && sizeof(T) == sizeof(double);
  // A level's factors: FP64 those of k_adv_prep.  FP32 forms them from s(k),
  // s(k+1) and the metric (a plane less to read), for the second pass again:
  // what a level carries between the passes is then four registers instead of
  // five
  struct Fac {
    T cu, cd, dv, nz;
    bool up;  // of interface k+1: the cell below is upwind
  };
  struct Lev {
    T a, b, c, d;  // FP64: cu, cd, dv, nz.  FP32: zu, zd
    T s, sp;       // s(k), s(k+1)
    bool up;
  };
  const double *__restrict__ cup = kPre ? D.vcu + ij : nullptr;
  const double *__restrict__ cdp = kPre ? D.vcd + ij : nullptr;
  const double *__restrict__ dvp = kPre ? D.vdiv + ij : nullptr;
  const double *__restrict__ nzp = kPre ? D.vnz + ij : nullptr;
  auto load = [&](unsigned o) {
    Lev r{};
    r.sp = T(sp[o + PS]);
    if constexpr (kPre) {
      r.a = T(cup[o]); r.b = T(cdp[o]); r.c = T(dvp[o]); r.d = T(nzp[o]);
    } else {
      r.a = T(zup[o]); r.b = T(zdp[o]);
    }
    return r;
  };
  auto factors = [&](const Lev &r) {
    if constexpr (kPre) {
      return Fac{r.a, r.b, r.c, r.d, r.up};
    } else {
      const T cu = mul_r(r.s, r.a), cd = mul_r(r.sp, r.b);
      const bool up = nonneg(r.sp);
      return Fac{cu, cd, cu - cd, fma_r(r.sp, hdtrdz, up ? T(0.5) : T(-0.5)), up};
    }
  };
  T c0k[NF], c0p1[NF], c1m2[NF], c1m1[NF], f1k[NF], f2m[NF], d1p[NF], d1c[NF], d2p[NF], d2c[NF], n_c[NF];
  // the next level's loads, issued one level ahead
  Lev n_l = load(0);
#pragma unroll
  for (int n = 0; n < NF; ++n) {
    c0k[n] = src[n][0];
    c0p1[n] = src[n][PS];
    n_c[n] = src[n][2 * PS];
    c1m2[n] = c1m1[n] = f1k[n] = f2m[n] = d1p[n] = d2p[n] = d2c[n] = T(0);
    d1c[n] = c0k[n] - c0p1[n];
  }
  T sk = kPre ? T(0) : T(sp[0]);
  Lev l1{}, l2{};  // levels k-1, k-2
  // level k; every bound check is known to hold inside the column
  // (4 <= k <= kz-3), so the interior steps carry none
  auto step = [&](int k, auto interior) {
    constexpr bool I = decltype(interior)::value;
    const unsigned o = (unsigned)(k - 1) * PS;
    Lev l = n_l;
    T c0p2[NF];
#pragma unroll
    for (int n = 0; n < NF; ++n) c0p2[n] = (I || k + 2 <= kz) ? n_c[n] : T(0);
    if (I || k < kz) {
      n_l = load(o + PS);
      if (I || k + 3 <= kz) {
#pragma unroll
        for (int n = 0; n < NF; ++n) n_c[n] = src[n][o + 3 * PS];
      }
    }
    if constexpr (kPre) {
      l.up = nonneg(l.sp);  // zamu has s's sign
    } else {
      l.s = sk;
      sk = l.sp;
    }
    const Fac t = factors(l), t2 = factors(l2);
#pragma unroll
    for (int n = 0; n < NF; ++n) {
      const T d1n = c0p1[n] - c0p2[n];  // the next interface's difference, this one's upwind one
      T f1kp;
      if (I) f1kp = vflux_in<T>(t.nz, t.up, c0k[n], c0p1[n], d1p[n], d1c[n], d1n);
      else f1kp = k <= kz - 1 ? vflux<T>(t.nz, t.up, c0k[n], c0p1[n], d1p[n], d1c[n], d1n, k, kz) : T(0);
      const T c1k = vupdate<T>(c0k[n], f1k[n], f1kp, t.dv, t.cu, t.cd);
      const T d2n = c1m1[n] - c1k;
      if (I || k >= 3) {  // pass 2 at level m = k-2
        T f2n;
        if (I) f2n = vflux_in<T>(t2.nz, t2.up, c1m2[n], c1m1[n], d2p[n], d2c[n], d2n);
        else f2n = vflux<T>(t2.nz, t2.up, c1m2[n], c1m1[n], d2p[n], d2c[n], d2n, k - 2, kz);
        dst[n][o - 2 * PS] = vupdate<T>(c1m2[n], f2m[n], f2n, t2.dv, t2.cu, t2.cd);
        f2m[n] = f2n;
      }
      c0k[n] = c0p1[n]; c0p1[n] = c0p2[n];
      c1m2[n] = c1m1[n]; c1m1[n] = c1k;
      d1p[n] = d1c[n]; d1c[n] = d1n; d2p[n] = d2c[n]; d2c[n] = d2n;
      f1k[n] = f1kp;
    }
    l2 = l1; l1 = l;
  };
  using edge = std::integral_constant<bool, false>;
  using mid = std::integral_constant<bool, true>;
  const int k1 = min(3, kz), k2 = max(4, kz - 2);
  for (int k = 1; k <= k1; ++k) step(k, edge{});
#pragma unroll 4
  for (int k = 4; k < k2; ++k) step(k, mid{});
  for (int k = k2; k <= kz; ++k) step(k, edge{});
  // pass 2 at levels kz-1 (flux through interface kz) and kz (none above)
  const unsigned ot = (unsigned)(kz - 1) * PS;
  const Fac t1 = factors(l1), t2 = factors(l2);
#pragma unroll
  for (int n = 0; n < NF; ++n) {
    const T f2n = vflux<T>(t2.nz, t2.up, c1m2[n], c1m1[n], d2p[n], d2c[n], T(0), kz - 1, kz);
    dst[n][ot - PS] = vupdate<T>(c1m2[n], f2m[n], f2n, t2.dv, t2.cu, t2.cd);
    dst[n][ot] = vupdate<T>(c1m1[n], f2n, T(0), t1.dv, t1.cu, t1.cd);
  }
}

// grid: x = column tiles along j times the groups of NF fields (group fastest,
// so the blocks reading one column's s and metric run together), y = row
// tiles, z = member; block (vert_x, vert_y) columns along (j, i)
template <class R, class T, int NF>
__global__ void __launch_bounds__(256, vert_min_blocks<T, NF>())
    k_adv_vertical(const Dom<R> *__restrict__ doms, int ng, int set, int advoff,
                               const WorkItem *__restrict__ wl) {
  grid_begin();
  const WorkItem wi = wl ? wl[blockIdx.x]
                          : WorkItem{(int16_t)blockIdx.z, (int16_t)(blockIdx.x / (unsigned)ng),
                                     (int16_t)blockIdx.y, (int16_t)(blockIdx.x % (unsigned)ng)};
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const int f0 = wi.c * NF, nf = set == 0 ? n_table_r(D) : 2;
  if (f0 >= nf) return;  // a member with fewer species
  const int j = wi.a * (int)blockDim.x + (int)threadIdx.x + 1;
  const int i = (int)wi.b * (int)blockDim.y + (int)threadIdx.y + 1;
  if (j > D.g.jx - 1 || i > D.g.iy - 1) return;
  const int adv = (D.clk->adv_role + advoff) & 1;
  const size_t ij = D.g.at2(j, i);
  if constexpr (NF == 2) {
    if (f0 + 1 >= nf) {
      vertical_column<R, T, 1>(D, set, f0, adv, ij);
      return;
    }
  }
  vertical_column<R, T, NF>(D, set, f0, adv, ij);
}


// Meridional then zonal WAF at one level for a tile of nw rows, every field
// of the R table (:984-1038; ROTLLR :926-983).  Warp w owns row I0+w; lane l
// owns v consecutive columns of it.  The winds, Courant numbers and metric
// coefficients of the lane's points are formed once, in registers, and then
// for each field in turn: its halo tile (rows I0-2 .. I0+nw+1, landed by TMA,
// double-buffered) gives the meridional fluxes of the warp's row, shared
// with the row above through shared memory (the last warp also forms the
// flux of row I0+nw); the intermediate p0 follows; the zonal fluxes take
// their neighbours' p0 from the adjacent lanes by shuffles, and the result
// goes to the field's other buffer (the halo of other tiles still needs the
// old values).  A warp's range is 32*v columns, of which an inner tile writes
// the middle 32*v - 4 (hshape_writes); tiles overlap by four columns.
// Resident warps an SM the WAF tile kernels are compiled for; the register
// budget follows (65536 / (32 * warps) a thread).  FP32, moist 512x512x41, a
// step: 64-column tiles at 40 warps (48 registers) 0.378 ms, at 32 0.434;
// 128-column tiles at 32 warps 0.351, at 24 0.394, at 40 (spilled) 0.471.
// The increment form at 32 warps (64 registers) 0.223 and 0.250 at 40 warps;
// in 128-column tiles at 16 warps (128 registers) 0.267, at 24 0.313.  FP64
// at 16 warps (108 registers): the FP64 pipe is the bound.
#ifndef MLC_HWAF_WARPS
#define MLC_HWAF_WARPS 40
#endif
#ifndef MLC_HWAF_WARPS_4
#define MLC_HWAF_WARPS_4 32
#endif
#ifndef MLC_HWAF_WARPS_D
#define MLC_HWAF_WARPS_D 16
#endif
#ifndef MLC_HINC_WARPS
#define MLC_HINC_WARPS 32
#endif
#ifndef MLC_HINC_WARPS_4
#define MLC_HINC_WARPS_4 16
#endif
template <class R>
constexpr int waf_min_blocks(int warps, int nw) {
  return warps / nw > 1 ? warps / nw : 1;
}
template <class R, int V, int NW>
__global__ void __launch_bounds__(32 * NW, waf_min_blocks<R>(sizeof(R) == sizeof(float)
                                                                   ? (V == 4 ? MLC_HWAF_WARPS_4 : MLC_HWAF_WARPS)
                                                                   : MLC_HWAF_WARPS_D, NW))
    k_adv_horizontal(const Dom<R> *__restrict__ doms,
                                                           int tiles_j, int uvoff, int advoff,
    const WorkItem *__restrict__ wl) {
  grid_begin();
  using T = R;
  constexpr int W = 32 * V;       // columns of a warp's range
  constexpr int S = W - 4;        // columns from a tile to the next (hshape_writes)
  constexpr unsigned kBox = (unsigned)((NW + 4) * W * sizeof(T));
  constexpr unsigned kBuf = (kBox + 127u) / 128u * 128u;
  constexpr int kStages = 4;  // halo tiles in flight: the next three fields land while one is used
  constexpr int shape = V == 1 ? (NW == 8 ? 0 : 3) : V == 2 ? (NW == 8 ? 1 : 2) : 4;
  static_assert(hshape((int)sizeof(T), shape).v == V && hshape((int)sizeof(T), shape).nw == NW,
                "tile shape table");
  __shared__ __align__(128) unsigned char wzraw[kStages][kBuf];  // TMA destinations
  __shared__ __align__(16) T zp_s[2][NW + 1][W];           // meridional fluxes, rows I0 .. I0+NW
  __shared__ __align__(8) uint64_t mbar[kStages];
  __shared__ const T *cur_s[kMaxFields];                   // each field's current and other half
  __shared__ T *out_s[kMaxFields];
  // grid: x = tiles along j and i, y = level, z = member
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const int k = wi.c + 1;
  const Geom g = D.g;
  const int jx = g.jx, iy = g.iy;
  if (k > g.kz) return;
  const int bj = wi.a, bi = wi.b;
  const int ob = bj * S;        // column offset (j - 1) of the range's first column
  const int I0 = bi * NW + 1;
  if (bj >= hshape_tiles(V, jx) || I0 > iy - 1) return;
  const Scal &c = D.c;
  const Stat<R> &sa = D.sa;
  const int uv = (D.clk->uv_role + uvoff) & 1, adv = (D.clk->adv_role + advoff) & 1;
  const int lane = (int)(threadIdx.x & 31u), wp = (int)(threadIdx.x >> 5);
  const int tid = (int)threadIdx.x;
  const int i = I0 + wp;
  const int e0 = ob + V * lane;                  // column offset of the lane's first column
  const bool inrow = e0 >= 0 && e0 + V <= g.P;   // the lane's columns lie inside a row
  const unsigned P = (unsigned)g.P;
  const unsigned ko = (unsigned)(k - 1) * (unsigned)g.PS;  // a field stays below 2^31 elements
  const T *__restrict__ uk = D.u[uv] + ko;
  const T *__restrict__ vk = D.v[uv] + ko;
  const T dta = pick<T>(c.dtstepa, c.dtstepaf);
  const T dtr = dta * pick<T>(c.rdx, c.rdxf);
  const bool rot = c.lrotllr != 0;
  const int nf = n_table_r(D);
  const char *tmaps = static_cast<const char *>(D.tmap) + (size_t)shape * kTmapSlots * kTmapBytes;
  auto tile = [&](int b) { return reinterpret_cast<T(*)[W]>(wzraw[b]); };
  auto issue = [&](int fld, int b) {  // one thread: the halo tile of field fld into buffer b
    fence_proxy_async();
    mbar_expect_tx(&mbar[b], kBox);
    tma_load_3d(wzraw[b], tmaps + (size_t)fld * kTmapBytes, ob, I0 - 3, k - 1, &mbar[b]);
  };
  if (tid == 0) {
    for (int q = 0; q < kStages; ++q) mbar_init(&mbar[q], 1);
    fence_mbar_init();
  }
  if (tid < nf) {
    const T *cur0;
    T *out0, *wz0;
    field_t<R, T>(D, 0, tid, adv, cur0, out0, wz0);
    cur_s[tid] = cur0 + ko;
    out_s[tid] = out0 + ko;
  }
  __syncthreads();
  if (D.stall_polls > 0) {
    // test hook: wait on a barrier that no copy completes (none is issued
    // yet), give up after the member's poll count and record the fault the
    // way the tile waits below do; the block leaves with nothing in flight
    const bool landed = mbar_wait_polls(&mbar[0], 0u, D.stall_polls);
    if (__syncthreads_or(!landed) && tid == 0) atomicOr(&D.clk->fault, 1);
    return;
  }
  if (tid == 0)
    for (int q = 0; q < kStages && q < nf; ++q) issue(q, q);

  // ---- the lane's coefficients (while the first tiles land) ----
  int jq[V];
#pragma unroll
  for (int q = 0; q < V; ++q) jq[q] = e0 + q + 1;
  const bool rowM = i >= 2 && i <= iy - 1;  // meridional flux rows
  const bool rowP = i >= 2 && i <= iy - 2;  // p0, zonal flux and update rows
  const bool okM = inrow && rowM, okP = inrow && rowP;
  // The fluxes of row I0+NW (the tile's north face): with two columns a lane
  // the last two warps take 32 columns each, one a lane, so that no warp
  // forms more than three flux rows' worth before the block barrier (the
  // last warp alone would form four); with one column a lane the last warp
  // takes them.  ec0 is the range column of the lane's first one there.
  constexpr int VE = NW >= V ? 1 : V;
  const bool eWarp = VE == 1 ? wp >= NW - V : wp == NW - 1;
  const int ec0 = VE == 1 ? (wp - (NW - V)) * 32 + lane : V * lane;
  const int eE0 = ob + ec0;
  // Courant numbers of the faces south of the lane's points, of row I0+NW and
  // west of the points, as upwind flags (zamu > 0) and -zmih
  bool upy[V], upe[VE], upx[V];
  T nzy[V], nze[VE], nzx[V];
  {
    T a[V], b[V];
    ld_row<T, V>(a, vk, e0, i, P, okM);
    ld_row<T, V>(b, sa.msfv, e0, i, P, okM && !rot);
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const T z = mul_r(rot ? a[q] : mul_r(a[q], b[q]), dtr);
      upy[q] = positive(z);
      nzy[q] = waf_nz<T>(z, upy[q]);
    }
    const int ie = I0 + NW;
    const bool okE = eWarp && eE0 >= 0 && eE0 + VE <= g.P && ie >= 2 && ie <= iy - 1;
    T ae[VE], be[VE];
    ld_row<T, VE>(ae, vk, eE0, ie, P, okE);
    ld_row<T, VE>(be, sa.msfv, eE0, ie, P, okE && !rot);
#pragma unroll
    for (int q = 0; q < VE; ++q) {
      const T z = mul_r(rot ? ae[q] : mul_r(ae[q], be[q]), dtr);
      upe[q] = positive(z);
      nze[q] = waf_nz<T>(z, upe[q]);
    }
  }
  // the faces' winds times dt/dx and the metric factors of the cell between
  // them (cs, cn; cw, ce) and the divergence factors (dvy, dvx), with
  // a = dt/dx*fmz*m^2 (rotated pole: *m).  rfmzu on the south and north faces
  // as in the reference (Main/mod_moloch.F90:1000-1001).
  T cs[V], cn[V], dvy[V], cw[V], ce[V], dvx[V];
  {
    T fz[V], vi[V], vn[V], ri[V], rn[V], fi[V], fn[V], mf[V], ui[V], rw[V], msu[V];
    ld_row<T, V>(fz, sa.fmz + ko, e0, i, P, okP);
    ld_row<T, V>(vi, vk, e0, i, P, okP);
    ld_row<T, V>(vn, vk, e0, i + 1, P, okP);
    ld_row<T, V>(ri, sa.rmv, e0, i, P, okP);
    ld_row<T, V>(rn, sa.rmv, e0, i + 1, P, okP);
    ld_row<T, V>(fi, (rot ? sa.rfmzv : sa.rfmzu) + ko, e0, i, P, okP);
    ld_row<T, V>(fn, (rot ? sa.rfmzv : sa.rfmzu) + ko, e0, i + 1, P, okP);
    ld_row<T, V>(mf, rot ? sa.msfx : sa.mx2, e0, i, P, okP);
    ld_row<T, V>(ui, uk, e0, i, P, okP);
    ld_row<T, V>(rw, sa.rmu, e0, i, P, okP && !rot);
    ld_row<T, V>(msu, sa.msfu, e0, i, P, okP);
    T fw[V], fe[V], ue[V], re[V];
    ld_row<T, V>(fw, sa.rfmzu + ko, e0, i, P, okP);
    next_col<T, V>(fe, fw);
    next_col<T, V>(ue, ui);
    next_col<T, V>(re, rw);
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const T a = mul_r(dtr, mul_r(fz[q], mf[q]));
      cs[q] = mul_r(mul_r(vi[q], rot ? mul_r(fi[q], ri[q]) : fi[q]), a);
      cn[q] = mul_r(mul_r(vn[q], rot ? mul_r(fn[q], rn[q]) : fn[q]), a);
      cw[q] = mul_r(mul_r(ui[q], fw[q]), a);
      ce[q] = mul_r(mul_r(ue[q], fe[q]), a);
      dvy[q] = rot ? cn[q] - cs[q] : fma_r(cn[q], rn[q], -mul_r(cs[q], ri[q]));
      dvx[q] = rot ? ce[q] - cw[q] : fma_r(ce[q], re[q], -mul_r(cw[q], rw[q]));
      const T z = mul_r(mul_r(ui[q], msu[q]), dtr);
      upx[q] = positive(z);
      nzx[q] = waf_nz<T>(z, upx[q]);
    }
  }
  // rows of the halo tile (global row r at tile row r - I0 + 2) the upwind
  // differences use, with the reference's clamps ih = min(i+1, imax),
  // ihm1 = max(ih-1, imin)
  auto mrows = [&](int r, int &ta, int &tb, int &tc) {
    ta = max(r - 2, 1) - I0 + 2;
    const int rb = min(r + 1, iy - 1);
    tb = rb - I0 + 2;
    tc = max(rb - 1, 1) - I0 + 2;
  };
  int tA, tB, tC, eA, eB, eC;
  mrows(i, tA, tB, tC);
  mrows(I0 + NW, eA, eB, eC);
  // columns the lane may write, and among them those it updates (the ring
  // keeps its values)
  bool wv[V], rv[V];
  bool wall = true;
#pragma unroll
  for (int q = 0; q < V; ++q) {
    wv[q] = inrow && i <= iy - 1 && hshape_writes(V, V * lane + q, ob, jx);
    rv[q] = rowP && jq[q] >= 2 && jq[q] <= jx - 2;
    wall = wall && wv[q];
  }
  const bool rowin = inrow && i <= iy - 1;

  for (int f = 0; f < nf; ++f) {
    const T *pp = cur_s[f];
    T *out = out_s[f];
    // the field's old values at the lane's points, in flight during the
    // meridional pass
    T ppk[V];
    ld_row<T, V>(ppk, pp, e0, i, P, rowin);
    const int b = f % kStages;
    const bool landed = mbar_wait_bounded(&mbar[b], (unsigned)((f / kStages) & 1));
    T(*wt)[W] = tile(b);
    T(*zp)[W] = zp_s[f & 1];
    // meridional fluxes per unit wind: j in jce, i in ici1..ice2 (elsewhere
    // they are not used)
    T wzi[V];
    {
      T wa[V], wA[V], wB[V], wC[V], x[V];
      ld_vec<T, V>(wa, &wt[i - I0 + 1][V * lane]);
      ld_vec<T, V>(wzi, &wt[i - I0 + 2][V * lane]);
      ld_vec<T, V>(wA, &wt[tA][V * lane]);
      ld_vec<T, V>(wB, &wt[tB][V * lane]);
      ld_vec<T, V>(wC, &wt[tC][V * lane]);
#pragma unroll
      for (int q = 0; q < V; ++q) {
        const bool up = upy[q];
        x[q] = waf_g<T>(nzy[q], up ? wa[q] : wzi[q], wzi[q] - wa[q], (up ? wa[q] : wB[q]) - (up ? wA[q] : wC[q]));
      }
      st_vec<T, V>(&zp[wp][V * lane], x);
      if (eWarp) {
        T xa[VE], xc[VE], eA_[VE], eB_[VE], eC_[VE], xe[VE];
        ld_vec<T, VE>(xa, &wt[NW + 1][ec0]);
        ld_vec<T, VE>(xc, &wt[NW + 2][ec0]);
        ld_vec<T, VE>(eA_, &wt[eA][ec0]);
        ld_vec<T, VE>(eB_, &wt[eB][ec0]);
        ld_vec<T, VE>(eC_, &wt[eC][ec0]);
#pragma unroll
        for (int q = 0; q < VE; ++q) {
          const bool up = upe[q];
          xe[q] = waf_g<T>(nze[q], up ? xa[q] : xc[q], xc[q] - xa[q],
                           (up ? xa[q] : eB_[q]) - (up ? eA_[q] : eC_[q]));
        }
        st_vec<T, VE>(&zp[NW][ec0], xe);
      }
    }
    if (__syncthreads_or(!landed)) {
      if (tid == 0) {
        atomicOr(&D.clk->fault, 1);
        // let copies still in flight land before the shared memory is released
        for (int g2 = f; g2 < f + kStages && g2 < nf; ++g2)
          mbar_wait_bounded(&mbar[g2 % kStages], (unsigned)((g2 / kStages) & 1));
      }
      return;
    }
    // buffer b is read for the last time above: fetch the field kStages on
    if (tid == 0 && f + kStages < nf) issue(f + kStages, b);
    // p0(j,i): j in jce, i in ici
    T p0[V];
    {
      T ys[V], yn[V];
      ld_vec<T, V>(ys, &zp[wp][V * lane]);
      ld_vec<T, V>(yn, &zp[wp + 1][V * lane]);
#pragma unroll
      for (int q = 0; q < V; ++q) p0[q] = waf_update<T>(wzi[q], ys[q], cs[q], yn[q], cn[q], dvy[q], ppk[q]);
    }
    // zonal fluxes zpbw(j,i): j in jci1..jce2, i in ici; p0 at range
    // columns c-2 .. c+1 (the lane's own, two from the lane to the west, one
    // from the lane to the east)
    T pw1 = __shfl_up_sync(0xffffffffu, p0[V - 1], 1);
    auto p0at = [&](int q) -> T {  // p0 of lane column q, q in -1 .. V-1
      return q < 0 ? pw1 : p0[q];
    };
    // differences p0(c) - p0(c-1) at the lane's columns, and those of the
    // columns either side from the neighbouring lanes: a column's den is the
    // num of its neighbours (upwind the one to the west, downwind the east)
    T dq[V];
#pragma unroll
    for (int q = 0; q < V; ++q) dq[q] = p0at(q) - p0at(q - 1);
    const T dw = __shfl_up_sync(0xffffffffu, dq[V - 1], 1);
    const T de = __shfl_down_sync(0xffffffffu, dq[0], 1);
    auto dat = [&](int q) -> T { return q < 0 ? dw : q >= V ? de : dq[q]; };
    T zx[V];
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const int j = jq[q];
      const bool up = upx[q];
      const T a = p0at(q - 1), cq = p0at(q);
      // jhm1 = max(j-2, jmin) upwind; jh = min(j+1, jmax) downwind:
      // upwind a - p0(jhm1), which is a - a at j = 2; downwind p0(jh) - p0(jh-1)
      const T num = up ? (j == 2 ? self_diff<T>(a) : dat(q - 1)) : (j == jx - 1 ? dq[q] : dat(q + 1));
      zx[q] = waf_g<T>(nzx[q], up ? a : cq, dq[q], num);
    }
    T zxe[V];
    next_col<T, V>(zxe, zx);
    // result: interior update, ring copied
    T res[V];
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const T x = waf_update<T>(p0[q], zx[q], cw[q], zxe[q], ce[q], dvx[q], ppk[q]);
      res[q] = rv[q] ? x : ppk[q];
    }
    if (wall) {
      st_vec<T, V>(out + (unsigned)e0 + (unsigned)(i - 1) * P, res);
    } else if (rowin) {
#pragma unroll
      for (int q = 0; q < V; ++q)
        if (wv[q]) out[(unsigned)(e0 + q) + (unsigned)(i - 1) * P] = res[q];
    }
  }
}

// Species that are not advected (ipptls = 0: qx(iqfrst:nqx)) keep their
// values when the advected fields move to the other half of their pairs.
template <class R, int LV>
__global__ void k_species_copy(const Dom<R> *__restrict__ doms, int advoff, int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const Pt q = point_at<LV>(wi, 1, 1);
  if (D.c.ipptls > 0 || q.j > g.jx - 1 || q.i > g.iy - 1 || q.k > g.kz) return;
  const int adv = (D.clk->adv_role + advoff) & 1;
  const size_t F = g.field3();
#pragma unroll
  for (int k = q.k; k < q.k + LV && k <= g.kz; ++k) {
    const size_t o = g.at(q.j, q.i, k);
    for (int n = 1; n < g.nqx; ++n) D.qx[adv ^ 1][o + (size_t)n * F] = D.qx[adv][o + (size_t)n * F];
  }
}

// :809-825
template <class R, int LV>
__global__ void k_adv_curvature(const Dom<R> *__restrict__ doms, int advoff, int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active || !D.c.curvature) return;
  const Geom g = D.g;
  const Scal &c = D.c;
  const Stat<R> &sa = D.sa;
  const int adv = (D.clk->adv_role + advoff) & 1;
  R *__restrict__ ux = D.ux[adv];
  R *__restrict__ vx = D.vx[adv];
  const Pt q_ = point_at<LV>(wi, 2, 2);
  const int j = q_.j, k0 = q_.k;
  if (k0 > g.kz) return;
  const int i = q_.i;
  if (j > g.jx - 2 || i > g.iy - 2) return;
  const size_t ij = g.at2(j, i);
  const R dta = pick<R>(c.dtstepa, c.dtstepaf);
  R tanx, tany;
  if (c.lrotllr) {
    tanx = R(sa.slat[i - 1]) * sa.msfx[ij] * R(kRearthRad);
    tany = tanx;
  } else {
    tanx = (sa.msfu[ij - 1] - sa.msfu[ij]) * pick<R>(c.rdx, c.rdxf);
    tany = (sa.msfv[ij - (size_t)g.P] - sa.msfv[ij]) * pick<R>(c.rdx, c.rdxf);
  }
#pragma unroll
  for (int k = k0; k < k0 + LV && k <= g.kz; ++k) {
    const size_t o = ij + (size_t)(k - 1) * g.PS;
    R a = ux[o];
    const R b = vx[o];
    a = fma_r(mul_r(mul_r(a, b), tanx), dta, a);
    ux[o] = a;
    vx[o] = fma_r(-mul_r(mul_r(a, a), tany), dta, b);
  }
}

// uvxtouvstag :1477-1522 and htozstag :1461-1475
template <class R, int LV>
__global__ void k_adv_back(const Dom<R> *__restrict__ doms, int uvoff, int advoff, int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const int uv = (D.clk->uv_role + uvoff) & 1, adv = (D.clk->adv_role + advoff) & 1;
  const R *__restrict__ ux = D.ux[adv];
  const R *__restrict__ vx = D.vx[adv];
  const R *__restrict__ wx = D.wx[adv];
  R *__restrict__ u = D.u[uv];
  R *__restrict__ v = D.v[uv];
  R *__restrict__ w = D.w;
  const Pt q_ = point_at<LV>(wi, 1, 1);
  const int j = q_.j, k0 = q_.k;
  if (k0 > g.kz) return;
  const int i = q_.i;
  const int jx = g.jx, iy = g.iy, kz = g.kz;
  if (j > jx || i > iy) return;
  const size_t ij = g.at2(j, i), PS = g.PS, S = (size_t)g.P;
  const bool do_u = (j >= 2 && j <= jx - 1 && i >= 2 && i <= iy - 2);
  const bool do_v = (j >= 2 && j <= jx - 2 && i >= 2 && i <= iy - 1);
  const bool do_w = (j <= jx - 1 && i <= iy - 1);
#pragma unroll
  for (int k = k0; k < k0 + LV && k <= g.kz; ++k) {
    const size_t o = ij + (size_t)(k - 1) * PS;
    if (do_u) {
      R a;
      if (j == jx - 1) a = R(0.5) * (ux[o - 1] + ux[o]);
      else if (j == 2) a = R(0.5) * (ux[o] + ux[o - 1]);
      else a = interp4<R>(ux[o], ux[o - 1], ux[o + 1], ux[o - 2]);
      u[o] = a;
    }
    if (do_v) {
      R a;
      if (i == iy - 1) a = R(0.5) * (vx[o - S] + vx[o]);
      else if (i == 2) a = R(0.5) * (vx[o] + vx[o - S]);
      else a = interp4<R>(vx[o], vx[o - S], vx[o + S], vx[o - 2 * S]);
      v[o] = a;
    }
    if (do_w && k >= 2) {
      R a;
      if (k == 2) a = R(0.5) * (wx[o] + wx[o - PS]);
      else if (k == kz) a = R(0.5) * (wx[o] + wx[o - PS]);
      else a = interp4<R>(wx[o], wx[o - PS], wx[o + PS], wx[o - 2 * PS]);
      w[o] = a;
      if (D.c.tke) {
        // htozstag(tkex, tke) (Main/mod_moloch.F90:831-834)
        const R *__restrict__ tx = D.tkex[adv];
        if (k == 2 || k == kz) a = R(0.5) * (tx[o] + tx[o - PS]);
        else a = interp4<R>(tx[o], tx[o - PS], tx[o + PS], tx[o - 2 * PS]);
        D.tke[o] = a;
      }
    }
  }
}

// k_adv_back of a mixed member in lanes of four columns, as k_adv_prep_v4
// (moist 512x512x41: 57 us a step against 94)
template <class R, int LV>
__global__ void __launch_bounds__(128) k_adv_back_v4(const Dom<R> *__restrict__ doms, int uvoff, int advoff,
                                                     int tiles_j, const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const int jx = g.jx, iy = g.iy, kz = g.kz;
  const int e0 = ((int)wi.a * 32 + (int)threadIdx.x) * 4, i = (int)wi.b * 4 + (int)threadIdx.y + 1;
  const int k0 = (int)wi.c * LV + 1;
  // (no wind is written in the last column and row)
  if (e0 + 1 > jx - 1 || i > iy - 1 || k0 > kz) return;
  const int uv = (D.clk->uv_role + uvoff) & 1, adv = (D.clk->adv_role + advoff) & 1;
  const unsigned P = (unsigned)g.P, PS = (unsigned)g.PS, ij = (unsigned)e0 + (unsigned)(i - 1) * P;
  const float *__restrict__ ux = D.ux[adv] + ij;
  const float *__restrict__ vx = D.vx[adv] + ij;
  const float *__restrict__ wx = D.wx[adv] + ij;
  const float *__restrict__ tx = D.c.tke ? D.tkex[adv] + ij : nullptr;
  float *__restrict__ u = D.u[uv] + ij;
  float *__restrict__ v = D.v[uv] + ij;
  float *__restrict__ w = D.w + ij;
  float *__restrict__ tk = D.c.tke ? D.tke + ij : nullptr;
  const bool do_u = i >= 2 && i <= iy - 2, do_v = i >= 2;
  // store columns first .. n-1 (0-based) of a lane
  auto store = [&](float *p, const float (&x)[4], int first, int n) {
    if (e0 >= first && e0 + 4 <= n) {
      st_vec<float, 4>(p, x);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (e0 + q >= first && e0 + q < n) p[q] = x[q];
    }
  };
  float w0[4] = {}, w1[4] = {}, w2[4], w3[4] = {};  // wx at levels k-2 .. k+1
  unsigned o = (unsigned)(k0 - 1) * PS;
  if (k0 >= 3) ld_vec<float, 4>(w0, wx + o - 2 * PS);
  if (k0 >= 2) ld_vec<float, 4>(w1, wx + o - PS);
  ld_vec<float, 4>(w2, wx + o);
  for (int k = k0; k < k0 + LV && k <= kz; ++k, o += PS) {
    float x[4];
    if (do_u) {
      float a[7] = {};  // columns e0-2 .. e0+4
      float m[4];
      ld_vec<float, 4>(m, ux + o);
      if (e0 >= 2) {
        a[0] = (ux + o)[-2];  // (o may be 0: no unsigned o - 2)
        a[1] = (ux + o)[-1];
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) a[2 + q] = m[q];
      if (e0 + 4 <= jx - 2) a[6] = ux[o + 4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int j = e0 + q + 1;
        x[q] = j == 2 || j == jx - 1 ? interp2<float>(a[q + 1], a[q + 2])
                                     : interp4<float>(a[q + 2], a[q + 1], a[q + 3], a[q]);
      }
      store(u + o, x, 1, jx - 1);
    }
    if (do_v) {
      float a[4] = {}, b[4], c[4], d[4] = {};  // rows i-2 .. i+1
      if (i >= 3) ld_vec<float, 4>(a, vx + o - 2 * P);
      ld_vec<float, 4>(b, vx + o - P);
      ld_vec<float, 4>(c, vx + o);
      if (i <= iy - 2) ld_vec<float, 4>(d, vx + o + P);
      interp_vec(x, c, b, d, a, i == 2 || i == iy - 1);
      store(v + o, x, 1, jx - 2);
    }
    if (k < kz) ld_vec<float, 4>(w3, wx + o + PS);
    if (k >= 2) {
      interp_vec(x, w2, w1, w3, w0, k == 2 || k == kz);
      store(w + o, x, 0, jx - 1);
      if (tx) {
        // htozstag(tkex, tke) (Main/mod_moloch.F90:831-834)
        float a[4] = {}, b[4], c[4], d[4] = {};
        if (k >= 3) ld_vec<float, 4>(a, tx + o - 2 * PS);
        ld_vec<float, 4>(b, tx + o - PS);
        ld_vec<float, 4>(c, tx + o);
        if (k < kz) ld_vec<float, 4>(d, tx + o + PS);
        interp_vec(x, c, b, d, a, k == 2 || k == kz);
        store(tk + o, x, 0, jx - 1);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) { w0[q] = w1[q]; w1[q] = w2[q]; w2[q] = w3[q]; }
  }
}

// ---- increment form for the FP64 fields (theta_v, Exner) of a mixed member --
//
// The WAF update is linear in the advected field once the limiter regions
// are fixed, and the regions depend on differences only.  So every flux can
// be formed from values relative to a reference r:
//   F(a - r, c - r, num) = F(a, c, num) - 2*hvel*r,
// and a cell's update relative to its own value needs only neighbour
// differences and the cell's own increment, all small numbers that FP32
// carries to ~1e-7 of the increment (not of the field).  FP64 is left for the
// neighbour differences, for the terms where the scheme does not preserve a
// constant field (the model top of the vertical pass, where the flux through
// kz+1 is zero but s(kz+1) is not; non-uniform map factors in the horizontal
// passes) and for the final sum field + increment.  Fluxes are formed once
// per interface, relative to the cell below (south, west) of it, and moved to
// the other cell's reference by -2*hvel*(its value - the first cell's).

// Both vertical passes (Main/mod_moloch.F90:858-922) in increment form, one
// thread per column, streaming the levels upward like k_adv_vertical with
// pass 2 two levels behind pass 1.  e is the pass input's increment over the
// field (zero for pass 1), dzs(k) = field(k+1) - field(k).  The flux per unit
// s through interface k+1 is formed relative to cell k and moved to cell k+1
// by -dzs(k).  Writes the increment dz = (field after the passes) - field, as
// a double-float at the bottom and top cells, which carry a double-float
// constant part (no flux through levels 1 and kz+1, where s need not vanish);
// elsewhere its low part is zero and is neither written nor read.
__device__ __forceinline__ float vflux_inc(float nz, bool up, float em1, float ek, float ekp1,
                                           float ekp2, float dzm1, float dzk, float dzp1, int k,
                                           int kz) {
  const float a = dzk + ekp1;
  float num;
  if (up) num = k + 2 <= kz ? (ekp1 - ekp2) - dzp1 : 0.f;
  else num = k >= 2 ? (em1 - ek) - dzm1 : 0.f;
  return waf_g<float>(nz, up ? a : ek, ek - a, num);
}
// the cell update without the bottom/top constant parts; gb is the flux per
// unit s through interface k (relative to cell k-1), ga the one through k+1
__device__ __forceinline__ float vupdate_inc(float ek, float gb, float ga, float cu, float cd,
                                             float dzm1, int k, int kz) {
  const float fb = k >= 2 ? gb - dzm1 : 0.f;
  const float fa = k <= kz - 1 ? ga : 0.f;
  return fma_r(fa, cd, fma_r(-fb, cu, mul_r(cu - cd, ek)));
}

template <class R>
__global__ void k_adv_vertical_inc(const Dom<R> *__restrict__ doms, int advoff,
                                   const WorkItem *__restrict__ wl) {
  grid_begin();
  const WorkItem wi = wl ? wl[blockIdx.x]
                          : WorkItem{(int16_t)blockIdx.z, (int16_t)(blockIdx.x >> 1), (int16_t)blockIdx.y,
                                     (int16_t)(blockIdx.x & 1u)};
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const int f = wi.c;
  const int bj = wi.a;
  const Geom g = D.g;
  const int kz = g.kz;
  const int j = bj * (int)blockDim.x + (int)threadIdx.x + 1;
  const int i = (int)wi.b * (int)blockDim.y + (int)threadIdx.y + 1;
  if (j > g.jx - 1 || i > g.iy - 1) return;
  const Scal &c = D.c;
  const int adv = (D.clk->adv_role + advoff) & 1;
  const size_t F = g.field3();
  const size_t ij = g.at2(j, i);
  // double-float planes: offsets count floats of the hi plane
  const DF src0(f == 0 ? D.tetav[adv] : D.pai[adv], F);
  const DF dst0(D.wz_d[f], F);
  const DF src{src0.p + ij, F};
  const DF dst{dst0.p + ij, F};
  const R *__restrict__ sp = D.s + ij;
  const R *__restrict__ zup = D.sa.zrfmu + ij;
  const R *__restrict__ zdp = D.sa.zrfmd + ij;
  const unsigned PS = (unsigned)g.PS;
  const float hdtrdz = -0.25f * (c.dtstepaf * c.rdzitaf);  // -1/2 of the factor of s in zamu

  // the bottom cell's and top cell's FP32 parts and double-float constant parts
  float eb32 = 0.f, et32 = 0.f;
  F2 hb{0.f, 0.f}, ht{0.f, 0.f};
  const F2 src1 = src.ld(0);
  // windows: field at k+1, dzs at k-3..k, pass-1 output at k-3..k-1, s at
  // k-2..k+1, metric at k-2..k-1, pass-1 flux at k (relative to k-1), pass-2
  // flux at k-2
  F2 xp1 = src.ld(PS);
  float dm3 = 0.f, dm2 = 0.f, dm1 = 0.f, dk = df_diff(xp1, src1);
  float e1m3 = 0.f, e1m2 = 0.f, e1m1 = 0.f;
  float sm2 = 0.f, sm1 = 0.f, sk = float(sp[0]);
  float zum2 = 0.f, zdm2 = 0.f, zum1 = 0.f, zdm1 = 0.f;
  float f1k = 0.f, f2m = 0.f;
  F2 n_x = src.ld(2 * PS);
  float n_s = float(sp[PS]), n_zu = float(zup[0]), n_zd = float(zdp[0]);
  // -zmih of an interface from its s
  auto nzof = [&](float s) { return fma_r(s, hdtrdz, s >= 0.f ? 0.5f : -0.5f); };
  // level k; the interior steps (4 <= k <= kz-3) carry no bound checks
  auto step = [&](int k, auto interior) {
    constexpr bool I = decltype(interior)::value;
    const unsigned o = (unsigned)(k - 1) * PS;
    const float skp1 = n_s, zuk = n_zu, zdk = n_zd;
    const F2 xp2 = n_x;  // field at k+2 (k+2 <= kz)
    if (I || k < kz) {
      n_s = float(sp[o + 2 * PS]);
      n_zu = float(zup[o + PS]);
      n_zd = float(zdp[o + PS]);
      if (I || k + 3 <= kz) n_x = src.ld(o + 3 * PS);
    }
    const float dp1 = I || k + 2 <= kz ? df_diff(xp2, xp1) : 0.f;  // dzs(k+1)
    // pass 1 (input increment zero)
    const int kk = I ? 4 : k, kzz = I ? 8 : kz;  // an interior level's checks hold
    const float f1kp = I || k <= kz - 1
                           ? vflux_inc(nzof(skp1), skp1 >= 0.f, 0.f, 0.f, 0.f, 0.f, dm1, dk, dp1, kk, kzz)
                           : 0.f;
    const float u1 = vupdate_inc(0.f, f1k, f1kp, mul_r(sk, zuk), mul_r(skp1, zdk), dm1, kk, kzz);
    float e1k = u1;
    if constexpr (!I) {
      if (k == kz) {
        et32 += u1;
        ht = df_add(ht, df_mul(src.ld(o), two_prod(-skp1, zdk)));
        e1k = et32 + df_f(ht);
      } else if (k == 1) {
        eb32 += u1;
        hb = df_add(hb, df_mul(src1, two_prod(sk, zuk)));
        e1k = eb32 + df_f(hb);
      }
    }
    if (I || k >= 3) {  // pass 2 at level m = k-2
      const int m = I ? 4 : k - 2;
      const float f2n = vflux_inc(nzof(sm1), sm1 >= 0.f, e1m3, e1m2, e1m1, e1k, dm3, dm2, dm1, m, kzz);
      const float u2 = vupdate_inc(e1m2, f2m, f2n, mul_r(sm2, zum2), mul_r(sm1, zdm2), dm3, m, kzz);
      if (!I && m == 1) {
        eb32 += u2;
        hb = df_add(hb, df_mul(src1, two_prod(sm2, zum2)));
        dst.st(o - 2 * PS, df_add_f(hb, eb32));
      } else {
        dst.p[o - 2 * PS] = e1m2 + u2;
      }
      f2m = f2n;
    }
    dm3 = dm2; dm2 = dm1; dm1 = dk; dk = dp1;
    xp1 = xp2;
    e1m3 = e1m2; e1m2 = e1m1; e1m1 = e1k;
    sm2 = sm1; sm1 = sk; sk = skp1;
    zum2 = zum1; zdm2 = zdm1; zum1 = zuk; zdm1 = zdk;
    f1k = f1kp;
  };
  using edge = std::integral_constant<bool, false>;
  using mid = std::integral_constant<bool, true>;
  const int k1 = min(3, kz), k2 = max(4, kz - 2);
  for (int k = 1; k <= k1; ++k) step(k, edge{});
#pragma unroll 4
  for (int k = 4; k < k2; ++k) step(k, mid{});
  for (int k = k2; k <= kz; ++k) step(k, edge{});
  // pass 2 at levels kz-1 and kz; dm3 = dzs(kz-2), dm2 = dzs(kz-1) now
  const unsigned ot = (unsigned)(kz - 1) * PS;
  const float f2n = vflux_inc(nzof(sm1), sm1 >= 0.f, e1m3, e1m2, e1m1, 0.f, dm3, dm2, dm1, kz - 1, kz);
  const float u2 = vupdate_inc(e1m2, f2m, f2n, mul_r(sm2, zum2), mul_r(sm1, zdm2), dm3, kz - 1, kz);
  dst.p[ot - PS] = e1m2 + u2;
  const float ut = vupdate_inc(e1m1, f2n, 0.f, mul_r(sm1, zum1), mul_r(sk, zdm1), dm2, kz, kz);
  et32 += ut;
  ht = df_add(ht, df_mul(src.ld(ot), two_prod(-sk, zdm1)));
  dst.st(ot, df_add_f(ht, et32));
}

// Meridional then zonal WAF (:984-1038; ROTLLR :926-983) in increment form
// for theta_v and Exner of a mixed member, at one level for a tile of nw rows,
// with the lane geometry of k_adv_horizontal: warp w owns row I0+w, lane l
// owns v consecutive columns, coefficients in registers, the meridional
// fluxes shared between rows through shared memory and the zonal neighbours
// taken from adjacent lanes.  pp is the field at the start of the advection
// step (double-float), dz its vertical increment; out = pp + dz + (meridional
// + zonal increments).  Fluxes are formed relative to the cell south (west)
// of the interface, from FP32 increments and neighbour differences.
template <class R, int V, int NW>
__global__ void __launch_bounds__(32 * NW, waf_min_blocks<R>(V == 4 ? MLC_HINC_WARPS_4 : MLC_HINC_WARPS, NW))
    k_adv_horizontal_inc(const Dom<R> *__restrict__ doms,
                                                               int tiles_j, int uvoff,
                                                               int advoff,
                                                               const WorkItem *__restrict__ wl) {
  grid_begin();
  constexpr int W = 32 * V, S = W - 4;
  constexpr unsigned kBox = (unsigned)((NW + 4) * W * 4);
  constexpr unsigned kBuf = (kBox + 127u) / 128u * 128u;
  constexpr int shape = V == 1 ? 0 : V == 2 ? 1 : 4;
  static_assert(hshape_inc(shape).v == V && hshape_inc(shape).nw == NW, "tile shape table");
  // per field: the halo tiles (rows I0-2 .. I0+NW+1) of pp hi, pp lo, dz hi,
  // dz lo, landed by TMA, all issued at the start
  __shared__ __align__(128) unsigned char tiles[2][4][kBuf];
  __shared__ __align__(16) float fy_s[2][NW + 1][W];  // meridional fluxes, rows I0 .. I0+NW
  __shared__ __align__(8) uint64_t mbar[2];
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const int k = wi.c + 1;
  const Geom g = D.g;
  const int jx = g.jx, iy = g.iy;
  if (k > g.kz) return;
  const int bj = wi.a, bi = wi.b;
  const int ob = bj * S;
  const int I0 = bi * NW + 1;
  if (bj >= hshape_tiles(V, jx) || I0 > iy - 1) return;
  const Scal &c = D.c;
  const Stat<R> &sa = D.sa;
  const int uv = (D.clk->uv_role + uvoff) & 1, adv = (D.clk->adv_role + advoff) & 1;
  const int lane = (int)(threadIdx.x & 31u), wp = (int)(threadIdx.x >> 5);
  const int i = I0 + wp;
  const int e0 = ob + V * lane;
  const bool inrow = e0 >= 0 && e0 + V <= g.P;
  const unsigned P = (unsigned)g.P;
  const unsigned ko = (unsigned)(k - 1) * (unsigned)g.PS;
  const size_t F = g.field3();
  const float *__restrict__ uk = D.u[uv] + ko;
  const float *__restrict__ vk = D.v[uv] + ko;
  const float dta = c.dtstepaf;
  const float dtr = dta * c.rdxf;
  const bool rot = c.lrotllr != 0;
  using T = float;
  const bool dlo = k == 1 || k == g.kz;  // elsewhere dz has no low part (k_adv_vertical_inc)
  const int tid = (int)threadIdx.x;
  if (tid == 0) {
    mbar_init(&mbar[0], 1);
    mbar_init(&mbar[1], 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (tid == 0) {
    const char *tm = static_cast<const char *>(D.tmap) + ((size_t)shape * kTmapSlots + kMaxFields) * kTmapBytes;
    for (int f = 0; f < 2; ++f) {
      const int ntile = dlo ? 4 : 3;
      mbar_expect_tx(&mbar[f], (unsigned)ntile * kBox);
      const int pslot = 4 * f + 2 * adv, dslot = 8 + 2 * f;
      const int slot[4] = {pslot, pslot + 1, dslot, dslot + 1};
      for (int q = 0; q < ntile; ++q)
        tma_load_3d(tiles[f][q], tm + (size_t)slot[q] * kTmapBytes, ob, I0 - 3, k - 1, &mbar[f]);
    }
  }

  int jq[V];
#pragma unroll
  for (int q = 0; q < V; ++q) jq[q] = e0 + q + 1;
  const bool rowM = i >= 2 && i <= iy - 1;
  const bool rowP = i >= 2 && i <= iy - 2;
  const bool okM = inrow && rowM, okP = inrow && rowP;
  const int ie = I0 + NW;
  const bool okE = wp == NW - 1 && inrow && ie >= 2 && ie <= iy - 1;
  // ---- coefficients, as in k_adv_horizontal ----
  T nzy[V], nze[V], nzx[V];
  bool upy[V], upe[V], upx[V], rv[V];
  {
    T a[V], b[V];
    ld_row<T, V>(a, vk, e0, i, P, okM);
    ld_row<T, V>(b, sa.msfv, e0, i, P, okM && !rot);
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const T z = mul_r(rot ? a[q] : mul_r(a[q], b[q]), dtr);
      upy[q] = z > 0.f;
      nzy[q] = waf_nz<T>(z, upy[q]);
    }
    ld_row<T, V>(a, vk, e0, ie, P, okE);
    ld_row<T, V>(b, sa.msfv, e0, ie, P, okE && !rot);
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const T z = mul_r(rot ? a[q] : mul_r(a[q], b[q]), dtr);
      upe[q] = z > 0.f;
      nze[q] = waf_nz<T>(z, upe[q]);
    }
  }
  // the faces' winds times the cell's metric factors (cs, cn; cw, ce) and the
  // map-factor terms that a constant field does not cancel (cy, cx)
  T cs[V], cn[V], cy[V], cw[V], ce[V], cx[V];
  bool cyf[V], cxf[V];
  {
    T fz[V], vi[V], vn[V], ri[V], rn[V], fi[V], fn[V], mf[V], ui[V], rw[V], msu[V];
    ld_row<T, V>(fz, sa.fmz + ko, e0, i, P, okP);
    ld_row<T, V>(vi, vk, e0, i, P, okP);
    ld_row<T, V>(vn, vk, e0, i + 1, P, okP);
    ld_row<T, V>(ri, sa.rmv, e0, i, P, okP);
    ld_row<T, V>(rn, sa.rmv, e0, i + 1, P, okP);
    ld_row<T, V>(fi, (rot ? sa.rfmzv : sa.rfmzu) + ko, e0, i, P, okP);
    ld_row<T, V>(fn, (rot ? sa.rfmzv : sa.rfmzu) + ko, e0, i + 1, P, okP);
    ld_row<T, V>(mf, rot ? sa.msfx : sa.mx2, e0, i, P, okP);
    ld_row<T, V>(ui, uk, e0, i, P, okP);
    ld_row<T, V>(rw, sa.rmu, e0, i, P, okP && !rot);
    ld_row<T, V>(msu, sa.msfu, e0, i, P, okP);
    T fw[V], fe[V], ue[V], re[V];
    ld_row<T, V>(fw, sa.rfmzu + ko, e0, i, P, okP);
    next_col<T, V>(fe, fw);
    next_col<T, V>(ue, ui);
    next_col<T, V>(re, rw);
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const T a = mul_r(dtr, mul_r(fz[q], mf[q]));
      cs[q] = mul_r(mul_r(vi[q], rot ? mul_r(fi[q], ri[q]) : fi[q]), a);
      cn[q] = mul_r(mul_r(vn[q], rot ? mul_r(fn[q], rn[q]) : fn[q]), a);
      cw[q] = mul_r(mul_r(ui[q], fw[q]), a);
      ce[q] = mul_r(mul_r(ue[q], fe[q]), a);
      cyf[q] = !rot && (ri[q] != 1.f || rn[q] != 1.f);
      cxf[q] = !rot && (rw[q] != 1.f || re[q] != 1.f);
      cy[q] = fma_r(cs[q], 1.f - ri[q], -mul_r(cn[q], 1.f - rn[q]));
      cx[q] = fma_r(cw[q], 1.f - rw[q], -mul_r(ce[q], 1.f - re[q]));
      const T z = mul_r(mul_r(ui[q], msu[q]), dtr);
      upx[q] = z > 0.f;
      nzx[q] = waf_nz<T>(z, upx[q]);
      rv[q] = okP && jq[q] >= 2 && jq[q] <= jx - 2;
    }
  }
  const bool rowin = inrow && i <= iy - 1;
  bool wv[V];
  bool wall = true;
#pragma unroll
  for (int q = 0; q < V; ++q) {
    const int cc = V * lane + q;
    wv[q] = rowin && hshape_writes(V, cc, ob, jx);
    wall = wall && wv[q];
  }
  // the meridional flux per unit wind through the south face of row r
  // (relative to pp(r-1)) from dz and pp differences of rows r-2 .. r+1; the
  // reference's clamps ih = min(r+1, imax), ihm1 = max(ih-1, imin)
  auto mflux = [&](T (&x)[V], const T (&nz)[V], const bool (&upr)[V], int r,
                   const T (&zm2)[V], const T (&zm1)[V], const T (&z0)[V], const T (&zp1)[V],
                   const T (&dym2)[V], const T (&dym1)[V], const T (&dy0)[V]) {
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const bool up = upr[q];
      const float cq = z0[q] + dym1[q];
      float num;
      if (up) num = r >= 3 ? (zm1[q] - zm2[q]) + dym2[q] : zm1[q] - zm1[q];
      else num = r <= iy - 2 ? (zp1[q] - z0[q]) + dy0[q] : (z0[q] - zm1[q]) + dym1[q];
      x[q] = waf_g<float>(nz[q], up ? zm1[q] : cq, cq - zm1[q], num);
    }
  };

  for (int f = 0; f < 2; ++f) {
    float *outh = reinterpret_cast<float *>(f == 0 ? D.tetav[adv ^ 1] : D.pai[adv ^ 1]);
    float (*fy)[W] = fy_s[f];
    const bool landed = mbar_wait_bounded(&mbar[f], 0u);
    const float(*tph)[W] = reinterpret_cast<const float(*)[W]>(tiles[f][0]);
    const float(*tpl)[W] = reinterpret_cast<const float(*)[W]>(tiles[f][1]);
    const float(*tzh)[W] = reinterpret_cast<const float(*)[W]>(tiles[f][2]);
    const float(*tzl)[W] = reinterpret_cast<const float(*)[W]>(tiles[f][3]);
    const int cl = V * lane;
    auto low_part = [&](T (&x)[V], const float *p) {
      if (dlo) {
        ld_vec<T, V>(x, p);
      } else {
#pragma unroll
        for (int q = 0; q < V; ++q) x[q] = 0.f;
      }
    };
    // rows i-2 .. i+1 (tile rows wp .. wp+3) of pp (hi, lo) and dz (rounded
    // to FP32); zero outside the cross points
    T ph[4][V], pl[4][V], zz[4][V], dzi_h[V], dzi_l[V];
#pragma unroll
    for (int rr = 0; rr < 4; ++rr) {
      ld_vec<T, V>(ph[rr], &tph[wp + rr][cl]);
      ld_vec<T, V>(pl[rr], &tpl[wp + rr][cl]);
      T zh[V], zl[V];
      ld_vec<T, V>(zh, &tzh[wp + rr][cl]);
      low_part(zl, &tzl[wp + rr][cl]);
#pragma unroll
      for (int q = 0; q < V; ++q) zz[rr][q] = zh[q] + zl[q];
      if (rr == 2) {
#pragma unroll
        for (int q = 0; q < V; ++q) { dzi_h[q] = zh[q]; dzi_l[q] = zl[q]; }
      }
    }
    // dy(r) = pp(r+1) - pp(r) for r = i-2, i-1, i
    T dy[3][V];
#pragma unroll
    for (int rr = 0; rr < 3; ++rr)
#pragma unroll
      for (int q = 0; q < V; ++q)
        dy[rr][q] = (ph[rr + 1][q] - ph[rr][q]) + (pl[rr + 1][q] - pl[rr][q]);
    {
      T x[V];
      mflux(x, nzy, upy, i, zz[0], zz[1], zz[2], zz[3], dy[0], dy[1], dy[2]);
      st_vec<T, V>(&fy[wp][V * lane], x);
    }
    if (wp == NW - 1) {  // the flux of row I0+NW: rows ie-2 .. ie+1 = i-1 .. i+2
      T h4[V], l4[V], zh[V], zl[V], z4[V], dy3[V];
      ld_vec<T, V>(h4, &tph[NW + 3][cl]);
      ld_vec<T, V>(l4, &tpl[NW + 3][cl]);
      ld_vec<T, V>(zh, &tzh[NW + 3][cl]);
      low_part(zl, &tzl[NW + 3][cl]);
#pragma unroll
      for (int q = 0; q < V; ++q) {
        z4[q] = zh[q] + zl[q];
        dy3[q] = (h4[q] - ph[3][q]) + (l4[q] - pl[3][q]);
      }
      T x[V];
      mflux(x, nze, upe, ie, zz[1], zz[2], zz[3], z4, dy[1], dy[2], dy3);
      st_vec<T, V>(&fy[NW][V * lane], x);
    }
    if (__syncthreads_or(!landed)) {
      if (tid == 0) {
        atomicOr(&D.clk->fault, 1);
        // let copies still in flight land before the shared memory is released
        mbar_wait_bounded(&mbar[f], 0u);
        if (f == 0) mbar_wait_bounded(&mbar[1], 0u);
      }
      return;
    }
    // p0 - pp: ey = dz + hy, hy the meridional increment
    T hy[V], ey[V];
    {
      T ys[V], yn[V];
      ld_vec<T, V>(ys, &fy[wp][V * lane]);
      ld_vec<T, V>(yn, &fy[wp + 1][V * lane]);
#pragma unroll
      for (int q = 0; q < V; ++q) {
        // the south flux moved to pp(i)
        float h = fma_r(ys[q] - dy[1][q], cs[q], -mul_r(yn[q], cn[q]));
        if (cyf[q]) h = fma_r(ph[2][q], cy[q], h);
        hy[q] = h;
        ey[q] = zz[2][q] + hy[q];
      }
    }
    // dx(j) = pp(j+1) - pp(j) at row i for the lane's columns; the east
    // neighbour's pp from the next lane
    T dx[V], dxw2, dxw1;
    {
      T eh[V], el[V];
      next_col<T, V>(eh, ph[2]);
      next_col<T, V>(el, pl[2]);
#pragma unroll
      for (int q = 0; q < V; ++q) dx[q] = (eh[q] - ph[2][q]) + (el[q] - pl[2][q]);
      dxw2 = __shfl_up_sync(0xffffffffu, dx[V >= 2 ? V - 2 : 0], V >= 2 ? 1 : 2);
      dxw1 = __shfl_up_sync(0xffffffffu, dx[V - 1], 1);
    }
    const float ew2 = __shfl_up_sync(0xffffffffu, ey[V >= 2 ? V - 2 : 0], V >= 2 ? 1 : 2);
    const float ew1 = __shfl_up_sync(0xffffffffu, ey[V - 1], 1);
    const float ee1 = __shfl_down_sync(0xffffffffu, ey[0], 1);
    auto eyat = [&](int q) -> float {
      return q == -2 ? ew2 : q == -1 ? ew1 : q == V ? ee1 : ey[q < 0 ? 0 : q >= V ? V - 1 : q];
    };
    auto dxat = [&](int q) -> float {
      return q == -2 ? dxw2 : q == -1 ? dxw1 : dx[q < 0 ? 0 : q >= V ? V - 1 : q];
    };
    // zonal fluxes per unit wind at the lane's columns, relative to pp(j-1)
    T fx[V];
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const int j = jq[q];
      const bool up = upx[q];
      const float a = eyat(q - 1), c0 = eyat(q), cq = c0 + dxat(q - 1);
      float num;
      if (up) num = j >= 3 ? (a - eyat(q - 2)) + dxat(q - 2) : a - a;
      else num = j <= jx - 2 ? (eyat(q + 1) - c0) + dxat(q) : (c0 - a) + dxat(q - 1);
      fx[q] = waf_g<float>(nzx[q], up ? a : cq, cq - a, num);
    }
    T fxe[V];
    next_col<T, V>(fxe, fx);
    // result
    T rh[V], rl[V];
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const F2 ppk{ph[2][q], pl[2][q]};
      F2 x = ppk;
      if (rv[q]) {
        // the west flux moved to pp(j)
        float hx = fma_r(fx[q] - dxat(q - 1), cw[q], -mul_r(fxe[q], ce[q]));
        if (cxf[q]) hx = fma_r(ppk.hi, cx[q], hx);
        x = df_add_f(df_add(ppk, F2{dzi_h[q], dzi_l[q]}), hy[q] + hx);
      }
      rh[q] = x.hi;
      rl[q] = x.lo;
    }
    float *oh = outh + ko + (unsigned)(i - 1) * P;
    if (wall) {
      st_vec<T, V>(oh + (unsigned)e0, rh);
      st_vec<T, V>(oh + F + (unsigned)e0, rl);
    } else if (rowin) {
#pragma unroll
      for (int q = 0; q < V; ++q)
        if (wv[q]) {
          oh[(unsigned)(e0 + q)] = rh[q];
          oh[F + (unsigned)(e0 + q)] = rl[q];
        }
    }
  }
}

// grid of a point kernel over nj x ni points per level
inline dim3 pt_grid(const LaunchGeom &L, int nj, int ni, int &tiles_j) {
  tiles_j = (nj + L.col_x - 1) / L.col_x;
  if (L.wl_pt) return dim3((unsigned)L.n_pt, 1, 1);  // one block per work item
  const int ti = (ni + L.col_y - 1) / L.col_y;
  return dim3((unsigned)(tiles_j * ti), (unsigned)((L.kz + L.lv - 1) / L.lv), (unsigned)L.nmem);
}

}  // namespace

// grid of the four-column kernels over nj x ni points (128 x 4 tiles)
dim3 v4_grid(const LaunchGeom &L, int nj, int ni, int &tj) {
  tj = (nj + 127) / 128;
  const int ti = (ni + 3) / 4;
  return L.wl_v4 ? dim3((unsigned)L.n_v4, 1, 1)
                 : dim3((unsigned)(tj * ti), (unsigned)((L.kz + L.lv - 1) / L.lv), (unsigned)L.nmem);
}

template <class R>
void Launch<R>::adv_prep(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  if constexpr (sizeof(R) == sizeof(float)) {
    int tj;
    const dim3 grd = v4_grid(L, L.jx - 1, L.iy - 1, tj), b(32, 4);
    if (L.lv == 1) step_launch(L, k_adv_prep_v4<R, 1>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_v4);
    else step_launch(L, k_adv_prep_v4<R, 4>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_v4);
    return;
  } else {
  const dim3 b((unsigned)L.col_x, (unsigned)L.col_y);
  int tj;
  const dim3 grd = pt_grid(L, L.jx - 1, L.iy - 1, tj);
  if (L.lv == 1) step_launch(L, k_adv_prep<R, 1>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_pt);
  else step_launch(L, k_adv_prep<R, 4>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_pt);
  }
}

template <class R, class T>
void launch_vertical(const LaunchGeom &L, const Dom<R> *d, int nf, int set, int advoff,
                     cudaStream_t s) {
  // one thread per column: blocks of vert_x x vert_y columns along (j, i)
  const dim3 b((unsigned)L.vert_x, (unsigned)L.vert_y);
  const int ng = (nf + L.vert_nf - 1) / L.vert_nf;
  const dim3 grd = L.wl_vert ? dim3((unsigned)L.n_vert, 1, 1)
                             : dim3((unsigned)(((L.jx - 1 + L.vert_x - 1) / L.vert_x) * ng),
                                    (unsigned)((L.iy - 1 + L.vert_y - 1) / L.vert_y), (unsigned)L.nmem);
  if constexpr (sizeof(T) == sizeof(float)) {
    if (L.vert_nf == 2) {
      step_launch(L, k_adv_vertical<R, T, 2>, grd, b, 0, s, d, ng, set, advoff, L.wl_vert);
      return;
    }
  }
  step_launch(L, k_adv_vertical<R, T, 1>, grd, b, 0, s, d, ng, set, advoff, L.wl_vert);
}

template <class R, int V, int NW>
void launch_tile(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  const int tj = hshape_tiles(V, L.jx), ti = (L.iy - 1 + NW - 1) / NW;
  const dim3 grd = L.wl_h ? dim3((unsigned)L.n_h, 1, 1)
                          : dim3((unsigned)(tj * ti), (unsigned)L.kz, (unsigned)L.nmem);
  step_launch(L, k_adv_horizontal<R, V, NW>, grd, 32 * NW, 0, s, d, tj, uvoff, advoff, L.wl_h);
}

template <class R>
void launch_horizontal(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  constexpr int eb = (int)sizeof(R);
  switch (waf_tile(L)) {
    case 4:
      if constexpr (sizeof(R) == sizeof(float)) launch_tile<R, 4, hshape(4, 4).nw>(L, d, uvoff, advoff, s);
      break;
    case 1: launch_tile<R, hshape(eb, 1).v, hshape(eb, 1).nw>(L, d, uvoff, advoff, s); break;
    case 2: launch_tile<R, hshape(eb, 2).v, hshape(eb, 2).nw>(L, d, uvoff, advoff, s); break;
    case 3: launch_tile<R, hshape(eb, 3).v, hshape(eb, 3).nw>(L, d, uvoff, advoff, s); break;
    default: launch_tile<R, hshape(eb, 0).v, hshape(eb, 0).nw>(L, d, uvoff, advoff, s); break;
  }
}

template <class R>
void launch_vertical_inc(const LaunchGeom &L, const Dom<R> *d, int advoff, cudaStream_t s) {
  const dim3 b((unsigned)L.vert_x, (unsigned)L.vert_y);
  const dim3 grd = L.wl_vinc ? dim3((unsigned)L.n_vinc, 1, 1)
                             : dim3((unsigned)(((L.jx - 1 + L.vert_x - 1) / L.vert_x) * 2),
                                    (unsigned)((L.iy - 1 + L.vert_y - 1) / L.vert_y), (unsigned)L.nmem);
  step_launch(L, k_adv_vertical_inc<R>, grd, b, 0, s, d, advoff, L.wl_vinc);
}

template <class R, int V, int NW>
void launch_tile_inc(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  const int tj = hshape_tiles(V, L.jx), ti = (L.iy - 1 + NW - 1) / NW;
  const dim3 grd = L.wl_hinc ? dim3((unsigned)L.n_hinc, 1, 1)
                             : dim3((unsigned)(tj * ti), (unsigned)L.kz, (unsigned)L.nmem);
  step_launch(L, k_adv_horizontal_inc<R, V, NW>, grd, 32 * NW, 0, s, d, tj, uvoff, advoff, L.wl_hinc);
}

template <class R>
void launch_horizontal_inc(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff,
                           cudaStream_t s) {
  switch (hshape_inc(waf_tile_inc(L)).v) {
    case 4: launch_tile_inc<R, 4, hshape_inc(4).nw>(L, d, uvoff, advoff, s); break;
    case 2: launch_tile_inc<R, 2, hshape_inc(1).nw>(L, d, uvoff, advoff, s); break;
    default: launch_tile_inc<R, 1, hshape_inc(0).nw>(L, d, uvoff, advoff, s); break;
  }
}

template <class R>
void Launch<R>::adv_vertical(const LaunchGeom &L, const Dom<R> *d, int advoff, cudaStream_t s) {
  launch_vertical<R, R>(L, d, L.nadv_r, 0, advoff, s);
}

template <class R>
void Launch<R>::adv_horizontal(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff,
                               cudaStream_t s) {
  launch_horizontal<R>(L, d, uvoff, advoff, s);
}

// The FP64 fields of a mixed member (L.nadv_d = 2) use the increment form.
template <class R>
void Launch<R>::adv_vertical_inc(const LaunchGeom &L, const Dom<R> *d, int advoff, cudaStream_t s) {
  if constexpr (sizeof(R) == sizeof(float)) launch_vertical_inc<R>(L, d, advoff, s);
}

template <class R>
void Launch<R>::adv_horizontal_inc(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff,
                                   cudaStream_t s) {
  if constexpr (sizeof(R) == sizeof(float)) launch_horizontal_inc<R>(L, d, uvoff, advoff, s);
}

template <class R>
void Launch<R>::adv_species_copy(const LaunchGeom &L, const Dom<R> *d, int advoff, cudaStream_t s) {
  const dim3 b((unsigned)L.col_x, (unsigned)L.col_y);
  int tj;
  const dim3 grd = pt_grid(L, L.jx - 1, L.iy - 1, tj);
  if (L.lv == 1) step_launch(L, k_species_copy<R, 1>, grd, b, 0, s, d, advoff, tj, L.wl_pt);
  else step_launch(L, k_species_copy<R, 4>, grd, b, 0, s, d, advoff, tj, L.wl_pt);
}

template <class R>
void Launch<R>::adv_curvature(const LaunchGeom &L, const Dom<R> *d, int advoff, cudaStream_t s) {
  const dim3 b((unsigned)L.col_x, (unsigned)L.col_y);
  int tj;
  const dim3 grd = pt_grid(L, L.jx - 3, L.iy - 3, tj);
  if (L.lv == 1) step_launch(L, k_adv_curvature<R, 1>, grd, b, 0, s, d, advoff, tj, L.wl_pt);
  else step_launch(L, k_adv_curvature<R, 4>, grd, b, 0, s, d, advoff, tj, L.wl_pt);
}

template <class R>
void Launch<R>::adv_back(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  if constexpr (sizeof(R) == sizeof(float)) {
    int tj;
    const dim3 grd = v4_grid(L, L.jx - 1, L.iy - 1, tj), b(32, 4);
    if (L.lv == 1) step_launch(L, k_adv_back_v4<R, 1>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_v4);
    else step_launch(L, k_adv_back_v4<R, 4>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_v4);
    return;
  } else {
  const dim3 b((unsigned)L.col_x, (unsigned)L.col_y);
  int tj;
  const dim3 grd = pt_grid(L, L.jx, L.iy, tj);
  if (L.lv == 1) step_launch(L, k_adv_back<R, 1>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_pt);
  else step_launch(L, k_adv_back<R, 4>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_pt);
  }
}

template <class R>
cudaError_t Launch<R>::configure_advect() {
  return cudaSuccess;
}

template struct Launch<double>;
template struct Launch<float>;

}  // namespace mlc
