// mlc_end.cu -- the end of the MOLOCH step (Main/mod_moloch.F90:340-446):
// virtual temperature and temperature, lateral boundary conditions
// (boundary :448-529 with bdyval, motopnudge, morelax of Main/mod_bdycod.F90
// and the tracer ring/relaxation of Main/chemlib/mod_che_bdyco.F90),
// pressure, density and saturation diagnostics, surface pressure
// extrapolation, status_update with zero tendencies, the mass budget of
// Main/mod_massck.F90 and the NaN/Inf check on ps.
//
// The boundary clock lives on the device: bdyval blends with xbctime, then
// the reference advances it by dtsec (Main/mod_bdycod.F90:2653) before
// motopnudge and morelax blend again, so those read xbctime + dtsec; the last
// kernel of a step stores the advanced clock (end_advance, or the reduction in
// split steps and those that nudge spectrally).
#include <algorithm>

#include "mlc_kernels.cuh"
#include "mlc_scalar.cuh"

namespace mlc {

namespace {

// 1 + ep1*qv - condensate (Main/mod_moloch.F90:1608-1648), of the species in q
template <class R>
__device__ __forceinline__ R qfactor_of(const R (&q)[5], int ipptls) {
  const R f = fma_r(R(kEp1), q[0], R(1));
  if (ipptls > 1) return f - q[1] - q[2] - q[3] - q[4];
  if (ipptls == 1) return f - q[1];
  return f;
}
// species in the factor
__device__ __forceinline__ int qfactor_species(int ipptls) { return ipptls > 1 ? 5 : ipptls == 1 ? 2 : 1; }
template <class R>
__device__ __forceinline__ R qfactor(const R *qx, size_t o, size_t F, int ipptls) {
  R q[5] = {};
  const int nq = qfactor_species(ipptls);
  for (int n = 0; n < 5; ++n)
    if (n < nq) q[n] = qx[o + (size_t)n * F];
  return qfactor_of<R>(q, ipptls);
}
// The same factor for a mixed member as the exact double-float 1 + d, with
// only d = ep1*qv - condensate in FP32.  The step end divides t by qf and
// multiplies by it again after the relaxation changed qv: an FP32 qf's
// rounding (6e-8) cancels only where qv did not change, and would otherwise
// reach theta_v in the relaxation zone every step.
__device__ __forceinline__ F2 qfactor_df_of(const float (&q)[5], int ipptls) {
  float d = mul_r(float(kEp1), q[0]);
  if (ipptls > 1) d = d - q[1] - q[2] - q[3] - q[4];
  else if (ipptls == 1) d = d - q[1];
  return fast_two_sum(1.f, d);
}
__device__ __forceinline__ F2 qfactor_df(const float *qx, size_t o, size_t F, int ipptls) {
  float q[5] = {};
  const int nq = qfactor_species(ipptls);
  for (int n = 0; n < 5; ++n)
    if (n < nq) q[n] = qx[o + (size_t)n * F];
  return qfactor_df_of(q, ipptls);
}

// Boundary blends and relaxations.  An FP64 member evaluates the reference's
// expressions x0*b0 + x1*b1 and (1 - x)*f + x*fext.  In FP32 both carry a
// rounding that repeats every step - 1 - x and x0 are rounded once and for
// all - and the relaxation turns it into a steady forcing of order
// eps*f/x (1e-5 of the field in the inner rings, with a ring-to-ring pattern
// that the divergence picks up); the increment forms b0 + x1*(b1 - b0) and
// f + x*(fext - f) round only the small correction.
template <class R>
__device__ __forceinline__ R bdy_blend(R x0, R x1, R b0, R b1) {
  if constexpr (sizeof(R) == sizeof(float)) return fmaf(x1, b1 - b0, b0);
  else return __fma_rn(x0, b0, __dmul_rn(x1, b1));
}
template <class R>
__device__ __forceinline__ R bdy_relax_to(R f, R x, R fext) {
  if constexpr (sizeof(R) == sizeof(float)) return fmaf(x, fext - f, f);
  else return __fma_rn(R(1) - x, f, __dmul_rn(x, fext));
}

// bdyval, MOLOCH branch (Main/mod_bdycod.F90:1631-1860): the west and east
// columns (corners excluded), then the south and north rows (corners
// included).  Species without boundary data, w and TKE take their floor on
// inflow and the value of the point inside on outflow; for a row's first and
// last point that is the column's new value, which the thread forms itself, so
// every ring point is independent: one thread a point and level.  (A block a
// level with a barrier between columns and rows took 204 us a step for 32
// members of 128x128x30, whose 960 blocks waited on memory one after the
// other.)
constexpr int kRingThreads = 128;
template <class R>
__global__ void __launch_bounds__(kRingThreads) k_bdy_ring(const Dom<R> *__restrict__ doms, int uvoff,
                                                           int advoff) {
  grid_begin();
  const Dom<R> &D = doms[blockIdx.z];
  if (!D.active) return;
  const Geom g = D.g;
  const int jx = g.jx, iy = g.iy;
  const int k = (int)blockIdx.y + 1;
  if (k > g.kz) return;
  const int n0 = iy - 2, n1 = jx;  // points a side: columns i = 2..iy-1, rows j = 1..jx
  int e = (int)(blockIdx.x * kRingThreads + threadIdx.x);
  if (e >= 2 * (n0 + n1)) return;
  const bool column = e < 2 * n0;
  if (!column) e -= 2 * n0;
  const bool far = e >= (column ? n0 : n1);  // east, north
  if (far) e -= column ? n0 : n1;
  const Scal &c = D.c;
  const Bdy<R> &bd = D.bd;
  const Clock *clk = D.clk;
  const State<R> st = state_of(D, (clk->uv_role + uvoff) & 1, (clk->adv_role + advoff) & 1);
  const double xb = clk->xbctime;
  const double x1 = (xb + c.dt) * c.rtb;
  const double x0 = 1.0 - x1;
  const R rx0 = R(x0), rx1 = R(x1);
  const size_t PS = g.PS, F = g.field3(), ko = (size_t)(k - 1) * PS;
  auto blend = [&](const R *const *b, size_t o) { return bdy_blend<R>(rx0, rx1, b[0][o], b[1][o]); };
  // j and i of the ring point (cross points), of the point inside it, and of
  // the wind normal to the side (u at jn in a column, v at row in)
  int j, i, jin, iin, jn, in;
  if (column) {
    i = in = iin = e + 2;
    j = far ? jx - 1 : 1; jin = far ? jx - 2 : 2; jn = far ? jx : 1;
  } else {
    j = jn = jin = e + 1;
    i = far ? iy - 1 : 1; iin = far ? iy - 2 : 2; in = far ? iy : 1;
  }
  const size_t on = g.at2(jn, in) + ko;
  // the winds along the side reach one point further than the cross points
  if (column) {
    st.v[g.at2(j, i) + ko] = blend(bd.dvb, g.at2(j, i) + ko);
    if (i > iy - 2) return;
  } else {
    st.u[g.at2(j, i) + ko] = blend(bd.dub, g.at2(j, i) + ko);
    if (j > jx - 1) return;
  }
  const R *const *nb = column ? bd.dub : bd.dvb;
  const R wind = blend(nb, on);
  (column ? st.u : st.v)[on] = wind;
  const size_t ob = g.at2(j, i) + ko;
  if (k == 1) {
    const size_t o2 = g.at2(j, i);
    st.ps[o2] = bdy_blend<double>(x0, x1, bd.xpsb[0][o2], bd.xpsb[1][o2]);
  }
  // t and Exner: x0*b0 + x1*b1 (a mixed member: b0 + x1*(b1 - b0) in
  // double-float, the low part of t in wz[1])
  if constexpr (sizeof(R) == sizeof(float)) {
    const DF t0(bd.xtb[0], F), t1(bd.xtb[1], F), p0(bd.xpaib[0], F), p1(bd.xpaib[1], F);
    const F2 a = t0.ld(ob), b = p0.ld(ob);
    const F2 t = df_add_f(a, mul_r(float(x1), df_diff(t1.ld(ob), a)));
    st.t[ob] = t.hi;
    D.wz[1][ob] = t.lo;
    DF(st.pai, F).st(ob, df_add_f(b, mul_r(float(x1), df_diff(p1.ld(ob), b))));
  } else {
    st.t[ob] = bdy_blend<double>(x0, x1, bd.xtb[0][ob], bd.xtb[1][ob]);
    st.pai[ob] = bdy_blend<double>(x0, x1, bd.xpaib[0][ob], bd.xpaib[1][ob]);
  }
  st.qx[ob] = blend(bd.xqb, ob);
  if (c.present_qc) st.qx[ob + F] = blend(bd.xlb, ob);
  if (c.present_qi && c.ipptls > 1) st.qx[ob + 2 * F] = blend(bd.xib, ob);
  // the point inside; at a row's ends a column point, whose own value is its
  // floor or that of the point inside it
  const bool west = !column && j == 1, east = !column && j == jx - 1;
  const size_t oi = g.at2(west ? 2 : east ? jx - 2 : jin, iin) + ko;
  const size_t oc = g.at2(west ? 1 : jx, iin) + ko;  // u of that column point
  auto inflow_of = [&](R x, bool hi) { return hi ? x < R(0) : x > R(0); };
  const bool floor1 = inflow_of(wind, far);
  const bool floor2 = (west || east) && inflow_of(blend(bd.dub, oc), east);
  const bool floor = floor1 || floor2;
  for (int n = 1; n < g.nqx; ++n) {
    if ((c.present_qc && n == 1) || (c.present_qi && n == 2)) continue;
    const size_t of = (size_t)n * F;
    st.qx[ob + of] = floor ? R(qx_zero(n)) : st.qx[oi + of];
  }
  st.w[ob] = floor ? R(0) : st.w[oi];
  if (c.tke) {
    // Main/mod_bdycod.F90:1684-1695, 1742-1753, 1800-1811, 1858-1869: the floor
    // at the top interface, below it inflow by the winds of levels k and k-1
    if (k == 1) {
      st.tke[ob] = R(kTkeMin);
    } else {
      const bool f1 = inflow_of(wind + blend(nb, on - PS), far);
      const bool f2 = (west || east) && inflow_of(blend(bd.dub, oc) + blend(bd.dub, oc - PS), east);
      st.tke[ob + PS] = f1 || f2 ? R(kTkeMin) : st.tke[oi + PS];
    }
  }
  if (g.ntr) {
    const double cx1 = (xb + c.dt) / c.dtbdys;  // chem_bdyval_uncoupled
    const double cx0 = 1.0 - cx1;
    for (int n = 0; n < g.ntr; ++n) {
      const size_t of = (size_t)n * F;
      st.trac[ob + of] = bdy_blend<R>(R(cx0), R(cx1), bd.chib[0][ob + of], bd.chib[1][ob + of]);
    }
  }
}

// The step end's point pass, after the boundary ring: virtual temperature
// and temperature of dynamical_core :1121-1123 (tvirt_to_temp :1629-1648),
// then - with the boundary on - motopnudge (Main/mod_bdycod.F90:4049-4083)
// and morelax on every field (boundary, Main/mod_moloch.F90:478-497).  Both
// are per point, so one thread does both at its points and t goes from the
// first to the second in registers.  The ring (bdyval) runs before this pass
// although the reference's order is tvirt, bdyval, relaxation: the ring reads
// only boundary data and the interior values of qx, w and TKE, which the
// temperature pass does not write, and it writes only ring points, where
// this pass leaves t alone; tvirt at the ring points is recomputed by the
// status update.  The relaxation's clock has already moved by dtsec.
template <class R, int LV>
__global__ void k_end_relax(const Dom<R> *__restrict__ doms, int uvoff, int advoff, int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const Scal &c = D.c;
  const Stat<R> &sa = D.sa;
  const Bdy<R> &bd = D.bd;
  const Clock *clk = D.clk;
  const State<R> st = state_of(D, (clk->uv_role + uvoff) & 1, (clk->adv_role + advoff) & 1);
  const Pt q_ = point_at<LV>(wi, 1, 1);
  const int j = q_.j, k0 = q_.k;
  if (k0 > g.kz) return;
  const int i = q_.i;
  const int jx = g.jx, iy = g.iy;
  if (j > jx - 1 || i > iy - 1) return;
  const bool inner = j >= 2 && j <= jx - 2 && i >= 2 && i <= iy - 2;
  const size_t ij = g.at2(j, i), PS = g.PS, F = g.field3();
  // the relaxation's points: jci x ici (t and the cross fields), jdi x ici
  // (u), jci x idi (v); none without the boundary
  const bool bdy = c.apply_bdy != 0 && j >= 2 && i >= 2;
  const bool cr = bdy && j <= jx - 2 && i <= iy - 2;
  const bool up = bdy && i <= iy - 2;
  const bool vp = bdy && j <= jx - 2;
  const double xb = clk->xbctime + c.dtsec;
  const double x1 = (xb + c.dt) * c.rtb;
  const double x0 = 1.0 - x1;
  const double cx1 = (xb + c.dt) / c.dtbdys;
  const double cx0 = 1.0 - cx1;
  const R rx0 = R(x0), rx1 = R(x1);
  const double trtau = 1.0 / (2.0 * 3600.0);
  const double wrtau = 1.0 / (3600.0 / 4.0);
  const int nsp = c.nspgx;
  const int ibc = cr ? sa.ibnd_cr[ij] : -1;
  const int ibu = up ? sa.ibnd_ud[ij] : -1;
  const int ibv = vp ? sa.ibnd_vd[ij] : -1;
  auto blend = [&](const R *const *b, size_t o) { return bdy_blend<R>(rx0, rx1, b[0][o], b[1][o]); };
  auto relax = [&](R f, R fext, int ib, int k) {
    const R xf = sa.hefc_r[(size_t)(ib - 1) + (size_t)(k - 1) * nsp];
    return bdy_relax_to<R>(f, xf, fext);
  };
  const R xfn0 = pick<R>(trtau * c.dtsec, float(trtau * c.dtsec));
  // The temperature part's inputs of a level, loaded one level ahead: the
  // next level's loads are issued before this level's stores (which would
  // otherwise hold them back, the arrays being reachable through one
  // descriptor), so each thread keeps two levels' loads in flight.
  const int ipp = c.ipptls;
  const int nq = ipp > 1 ? 5 : ipp == 1 ? 2 : 1;
  struct TvIn {
    R th, pa, q[5];
    float thl, pal;  // a mixed member's low parts of theta_v and Exner
  };
  auto load_in = [&](size_t o, TvIn &x) {
    if constexpr (sizeof(R) == sizeof(float)) {
      const DF th(st.tetav, F), pa(st.pai, F);
      const F2 a = th.ld(o), b = pa.ld(o);
      x.th = a.hi; x.thl = a.lo; x.pa = b.hi; x.pal = b.lo;
    } else {
      x.th = R(st.tetav[o]); x.pa = R(st.pai[o]); x.thl = x.pal = 0.f;
    }
#pragma unroll
    for (int n = 0; n < 5; ++n) x.q[n] = n < nq ? st.qx[o + (size_t)n * F] : R(0);
  };
  TvIn cur, nxt;
  load_in(ij + (size_t)(k0 - 1) * PS, cur);
#pragma unroll
  for (int k = k0; k < k0 + LV && k <= g.kz; ++k) {
    const size_t o = ij + (size_t)(k - 1) * PS;
    if (k + 1 < k0 + LV && k + 1 <= g.kz) load_in(o + PS, nxt);
    // ---- tvirt and t (every cross point; t only inside the ring) ----
    F2 tdf{0.f, 0.f};  // a mixed member's double-float t
    R tr = R(0);       // an FP64 member's t
    if constexpr (sizeof(R) == sizeof(float)) {
      // t as a double-float through the step end: hi in t, lo in wz[1] (the
      // scratch is free until the next advection); status_update rebuilds
      // theta_v = t*qf/pai from it, so t's FP32 rounding never reaches theta_v
      const F2 tv = df_mul(F2{cur.th, cur.thl}, F2{cur.pa, cur.pal});
      st.tvirt[o] = df_f(tv);
      if (inner) {
        tdf = df_div(tv, qfactor_df_of(cur.q, ipp));
      } else if (!c.apply_bdy) {
        D.wz[1][o] = 0.f;  // (with the boundary on, the ring wrote it)
      }
    } else {
      const R tv = mul_r(cur.th, cur.pa);
      st.tvirt[o] = tv;
      if (inner) tr = divide<R>(tv, qfactor_of<R>(cur.q, ipp));
    }
    cur = nxt;
    // ---- motopnudge and morelax ----
    if (k == 2 && cr && c.top_nudge) {
      const size_t o2 = ij + PS;  // level 2 (w sponge, before the level's relaxation)
      const R xf = R(wrtau * c.dtsec);
      const R w2 = st.w[o2];
      const R fext = R(0) * w2;
      st.w[o2] = bdy_relax_to<R>(w2, xf, fext);
    }
    const bool nud = c.top_nudge && k <= c.nztop;
    R xfn;
    if constexpr (sizeof(R) == sizeof(float)) xfn = nud ? sa.tnudge_r[k - 1] * xfn0 : R(0);
    else xfn = nud ? R(sa.tnudge[k - 1] * trtau * c.dtsec) : R(0);
    // only nudged levels and the relaxation zone change anything
    if (up && (nud || ibu > 0)) {
      R f = st.u[o];
      if (nud) f = bdy_relax_to<R>(f, xfn, blend(bd.dub, o));
      if (ibu > 0) f = relax(f, blend(bd.dub, o), ibu, k);
      st.u[o] = f;
    }
    if (vp && (nud || ibv > 0)) {
      R f = st.v[o];
      if (nud) f = bdy_relax_to<R>(f, xfn, blend(bd.dvb, o));
      if (ibv > 0) f = relax(f, blend(bd.dvb, o), ibv, k);
      st.v[o] = f;
    }
    if (cr && (nud || ibc > 0)) {
      if constexpr (sizeof(R) == sizeof(float)) {
        // (1-x)*t + x*b as t + x*(b - t) on the double-float t
        const DF b0(bd.xtb[0], F), b1(bd.xtb[1], F);
        const F2 a = b0.ld(o);
        const F2 bt = df_add_f(a, mul_r(float(x1), df_diff(b1.ld(o), a)));
        if (nud) tdf = df_add_f(tdf, mul_r(xfn, df_diff(bt, tdf)));
        if (ibc > 0) {
          const float xf = sa.hefc_r[(size_t)(ibc - 1) + (size_t)(k - 1) * nsp];
          tdf = df_add_f(tdf, mul_r(xf, df_diff(bt, tdf)));
        }
      } else {
        const double bt = bdy_blend<double>(x0, x1, bd.xtb[0][o], bd.xtb[1][o]);
        if (nud) tr = bdy_relax_to<R>(tr, xfn, R(bt));
        if (ibc > 0) tr = relax(tr, R(bt), ibc, k);
      }
    }
    if (inner) {
      if constexpr (sizeof(R) == sizeof(float)) {
        st.t[o] = tdf.hi;
        D.wz[1][o] = tdf.lo;
      } else {
        st.t[o] = tr;
      }
    }
    if (!cr || ibc <= 0) continue;
    if constexpr (sizeof(R) == sizeof(float)) {
      // (1 - xf)*pai + xf*(b0 + x1*(b1 - b0)) as pai + xf*((b0 - pai) + x1*(b1 - b0))
      const float xf = sa.hefc_r[(size_t)(ibc - 1) + (size_t)(k - 1) * nsp];
      const DF pa(st.pai, F), b0(bd.xpaib[0], F), b1(bd.xpaib[1], F);
      const F2 pp = pa.ld(o), a = b0.ld(o);
      pa.st(o, df_add_f(pp, mul_r(xf, fmaf(float(x1), df_diff(b1.ld(o), a), df_diff(a, pp)))));
    } else {
      const double xf = sa.hefc[(size_t)(ibc - 1) + (size_t)(k - 1) * nsp];
      st.pai[o] = bdy_relax_to<double>(st.pai[o], xf, bdy_blend<double>(x0, x1, bd.xpaib[0][o], bd.xpaib[1][o]));
    }
    st.qx[o] = relax(st.qx[o], blend(bd.xqb, o), ibc, k);
    {
      // morelax_fraction with frac = 0 (:3962-3993)
      const R xf = sa.hefc_r[(size_t)(ibc - 1) + (size_t)(k - 1) * nsp];
      const R f = st.w[o];
      st.w[o] = bdy_relax_to<R>(f, xf, f * R(0));
    }
    if (c.ipptls > 0 && c.present_qc) st.qx[o + F] = relax(st.qx[o + F], blend(bd.xlb, o), ibc, k);
    if (c.ipptls > 1 && c.present_qi) st.qx[o + 2 * F] = relax(st.qx[o + 2 * F], blend(bd.xib, o), ibc, k);
    for (int n = 0; n < g.ntr; ++n) {
      const size_t on = o + (size_t)n * F;
      const R xf = sa.fcx_r[ibc - 1];
      const R fext = bdy_blend<R>(R(cx0), R(cx1), bd.chib[0][on], bd.chib[1][on]);
      st.trac[on] = bdy_relax_to<R>(st.trac[on], xf, fext);
    }
  }
}

// ---- spectral nudging (Main/mod_bdycod.F90:3898-3960, called from
// Main/mod_moloch.F90:499-506 after the relaxation) ----
// The reference projects the departure d = blend(b0,b1) - f of t, u and v
// onto km2 sine modes in x (sums over the field's interior columns jj), back
// to the grid, onto lm2 modes in y (sums over its interior rows ii) and back,
// and adds cnudge(k) times the result on jj x ii.  Only d on jj x ii enters,
// and the four passes factor into
//   sx(i,m) = sum_{j in jj} d(j,i) bvx(j,m)                 (k_spec_rows)
//   C(m,l)  = sum_{i in ii} sx(i,m) bvy(i,l)                (k_spec_modes)
//   G(i,m)  = sum_l C(m,l) bvy(i,l)                          (k_spec_modes)
//   f(j,i) += cnudge(k) sum_m bvx(j,m) G(i,m)                (k_spec_apply)
// per field, level and member.  Ranges: t jj = jci1..jci1 (the reference's
// call passes jci1 as both bounds), ii = ici; u jdi x ici; v jci x idi.
// The kernels run every step and return at once unless the interval is due.

// the step's boundary update is a spectral nudging step: tspectral + dtsec
// (the reference's tspectral after its increment) is a multiple of dtrad
__device__ __forceinline__ bool spectral_due(const Scal &c, const Clock *clk) {
  return c.spectral && (int)fmod(clk->tspectral + c.dtsec, c.dtrad) == 0;
}
struct SpecRange {
  int jj1, jj2, ii1, ii2;
};
__device__ __forceinline__ SpecRange spec_range(int f, const Geom &g) {
  if (f == 0) return {2, 2, 2, g.iy - 2};
  if (f == 1) return {2, g.jx - 1, 2, g.iy - 2};
  return {2, g.jx - 2, 2, g.iy - 1};
}

// Departure of field f (0 t, 1 u, 2 v) from the blended boundary data at o.
template <class R>
__device__ __forceinline__ R spec_departure(const Dom<R> &D, const State<R> &st, int f, size_t o,
                                            double x0, double x1) {
  const Bdy<R> &bd = D.bd;
  if (f == 0) {
    if constexpr (sizeof(R) == sizeof(float)) {
      const size_t F = D.g.field3();
      const DF b0(bd.xtb[0], F), b1(bd.xtb[1], F);
      const F2 a = b0.ld(o);
      const F2 bt = df_add_f(a, float(x1) * df_diff(b1.ld(o), a));
      return df_diff(bt, F2{st.t[o], D.wz[1][o]});
    } else {
      return bdy_blend<double>(x0, x1, bd.xtb[0][o], bd.xtb[1][o]) - st.t[o];
    }
  }
  const R *const *b = f == 1 ? bd.dub : bd.dvb;
  const R cur = f == 1 ? st.u[o] : st.v[o];
  return bdy_blend<R>(R(x0), R(x1), b[0][o], b[1][o]) - cur;
}

// sx(i, m) of one row: a warp per row i, lanes over j; grid (rows/8,
// kz*3, members), 256 threads.
template <class R>
__global__ void __launch_bounds__(256) k_spec_rows(const Dom<R> *__restrict__ doms, int uvoff, int advoff) {
  grid_begin();
  const Dom<R> &D = doms[blockIdx.z];
  if (!D.active) return;
  const Scal &c = D.c;
  const Clock *clk = D.clk;
  if (!spectral_due(c, clk)) return;
  const Geom g = D.g;
  const int k = (int)blockIdx.y / 3 + 1, f = (int)blockIdx.y % 3;
  if (k > g.kz) return;
  const SpecRange r = spec_range(f, g);
  const int lane = (int)threadIdx.x & 31;
  const int i = r.ii1 + (int)blockIdx.x * 8 + ((int)threadIdx.x >> 5);
  if (i > r.ii2) return;
  const State<R> st = state_of(D, (clk->uv_role + uvoff) & 1, (clk->adv_role + advoff) & 1);
  const double x1 = (clk->xbctime + c.dtsec + c.dt) * c.rtb, x0 = 1.0 - x1;
  const int km2 = c.km2;
  const R *bvx = D.sa.bvx;
  R acc[kMaxModes];
#pragma unroll
  for (int m = 0; m < kMaxModes; ++m) acc[m] = R(0);
  const size_t row = g.at2(1, i) + (size_t)(k - 1) * g.PS;
  for (int j = r.jj1 + lane; j <= r.jj2; j += 32) {
    const R dv = spec_departure(D, st, f, row + (size_t)(j - 1), x0, x1);
#pragma unroll
    for (int m = 0; m < kMaxModes; ++m)
      if (m < km2) acc[m] += dv * bvx[(size_t)m * g.jx + (j - 1)];
  }
  R mine = R(0);
#pragma unroll
  for (int m = 0; m < kMaxModes; ++m) {
    if (m < km2) {
      R v = acc[m];
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
      if (lane == m) mine = v;
    }
  }
  if (lane < km2)
    D.spec[((size_t)(f * g.kz + k - 1) * g.iy + (size_t)(i - 1)) * km2 + lane] = mine;
}

// C(m, l) in shared memory, then G(i, m) over sx in place; one block of 256
// threads per field, level and member.
template <class R>
__global__ void __launch_bounds__(256) k_spec_modes(const Dom<R> *__restrict__ doms) {
  grid_begin();
  const Dom<R> &D = doms[blockIdx.z];
  if (!D.active) return;
  const Scal &c = D.c;
  if (!spectral_due(c, D.clk)) return;
  const Geom g = D.g;
  const int k = (int)blockIdx.y / 3 + 1, f = (int)blockIdx.y % 3;
  if (k > g.kz) return;
  const SpecRange r = spec_range(f, g);
  const int km2 = c.km2, lm2 = c.lm2, ni = r.ii2 - r.ii1 + 1;
  const R *bvy = D.sa.bvy;
  R *sx = D.spec + (size_t)(f * g.kz + k - 1) * g.iy * km2;
  __shared__ R cm[kMaxModes * kMaxModes];
  for (int p = (int)threadIdx.x; p < km2 * lm2; p += (int)blockDim.x) {
    const int m = p / lm2, l = p % lm2;
    R a = R(0);
    for (int i = r.ii1; i <= r.ii2; ++i) a += sx[(size_t)(i - 1) * km2 + m] * bvy[(size_t)l * g.iy + (i - 1)];
    cm[p] = a;
  }
  __syncthreads();
  for (int p = (int)threadIdx.x; p < ni * km2; p += (int)blockDim.x) {
    const int i = r.ii1 + p / km2, m = p % km2;
    R a = R(0);
    for (int l = 0; l < lm2; ++l) a += cm[m * lm2 + l] * bvy[(size_t)l * g.iy + (i - 1)];
    sx[(size_t)(i - 1) * km2 + m] = a;
  }
}

// f(j,i,k) += cnudge(k) sum_m bvx(j,m) G(i,m) for t, u and v at one point
// (j, i from 2), LV levels per thread.
template <class R, int LV>
__global__ void k_spec_apply(const Dom<R> *__restrict__ doms, int uvoff, int advoff, int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Scal &c = D.c;
  const Clock *clk = D.clk;
  if (!spectral_due(c, clk)) return;
  const Geom g = D.g;
  const Pt q_ = point_at<LV>(wi, 2, 2);
  const int j = q_.j, i = q_.i, k0 = q_.k;
  if (k0 > g.kz || j > g.jx - 1 || i > g.iy - 1) return;
  const State<R> st = state_of(D, (clk->uv_role + uvoff) & 1, (clk->adv_role + advoff) & 1);
  const int km2 = c.km2;
  const R *bvx = D.sa.bvx + (j - 1);
  const size_t ij = g.at2(j, i);
  auto proj = [&](int f, int k) {
    const R *gg = D.spec + ((size_t)(f * g.kz + k - 1) * g.iy + (size_t)(i - 1)) * km2;
    R a = R(0);
    for (int m = 0; m < km2; ++m) a += bvx[(size_t)m * g.jx] * gg[m];
    return a;
  };
  const bool tp = j == 2 && i <= g.iy - 2, up = i <= g.iy - 2, vp = j <= g.jx - 2;
#pragma unroll
  for (int k = k0; k < k0 + LV && k <= g.kz; ++k) {
    const size_t o = ij + (size_t)(k - 1) * g.PS;
    const R cn = D.sa.cnudge[k - 1];
    if (tp) {
      if constexpr (sizeof(R) == sizeof(float)) {
        const F2 t = df_add_f(F2{st.t[o], D.wz[1][o]}, cn * proj(0, k));
        st.t[o] = t.hi;
        D.wz[1][o] = t.lo;
      } else {
        st.t[o] = st.t[o] + cn * proj(0, k);
      }
    }
    if (up) st.u[o] = st.u[o] + cn * proj(1, k);
    if (vp) st.v[o] = st.v[o] + cn * proj(2, k);
  }
}

// extrapolate_surface_pressure (:1592-1606) from the virtual temperatures and
// heights of the levels kz-1 and kz and the pressure of the lowest.
__device__ __forceinline__ double surface_pressure(double tv1, double tv2, double z1, double z2, double p2) {
  double lrt = div_d(tv1 - tv2, z1 - z2);
  if (lrt < -kGovcp) lrt = -kGovcp;
  else if (lrt > -0.005) lrt = __fma_rn(0.65, lrt, -0.35 * kLrate);
  const double tv = __fma_rn(__dmul_rn(-lrt, 0.5), z2, tv2);
  return __dmul_rn(p2, exp(div_d(__dmul_rn(kGovr, z2), tv)));
}
// The same of the interior column at ij, from t and q before status_update
// clamps q, and p at the lowest level (the expression k_end_cross stores).
template <class R>
__device__ __forceinline__ void ps_column(const Dom<R> &D, const State<R> &st, size_t ij) {
  const Geom &g = D.g;
  const Scal &c = D.c;
  const size_t PS = g.PS, F = g.field3();
  const int ipp = c.ipptls, kz = g.kz;
  // tvirt at kz-1, kz before the clamps: from the boundary's temp_to_tvirt,
  // or tetav*pai of dynamical_core when the boundary is off
  const size_t o1 = ij + (size_t)(kz - 2) * PS, o2 = ij + (size_t)(kz - 1) * PS;
  double tv1, tv2;
  if (c.apply_bdy) {
    tv1 = (double)mul_r(st.t[o1], qfactor(st.qx, o1, F, ipp));
    tv2 = (double)mul_r(st.t[o2], qfactor(st.qx, o2, F, ipp));
  } else {
    tv1 = (double)st.tvirt[o1];
    tv2 = (double)st.tvirt[o2];
  }
  R p2;
  if constexpr (sizeof(R) == sizeof(float)) p2 = exner_to_pressure_f(df_f(DF(st.pai, F).ld(o2)));
  else p2 = (R)exner_to_pressure(st.pai[o2]);
  st.ps[ij] = surface_pressure(tv1, tv2, D.sa.zeta[o1], D.sa.zeta[o2], (double)p2);
}

// ps of every interior column, for the split step and steps with spectral
// nudging (the reduction forms it in the others)
template <class R>
__global__ void k_end_ps(const Dom<R> *__restrict__ doms, int uvoff, int advoff) {
  grid_begin();
  const Dom<R> &D = doms[blockIdx.z];
  if (!D.active) return;
  const Geom g = D.g;
  const State<R> st = state_of(D, (D.clk->uv_role + uvoff) & 1, (D.clk->adv_role + advoff) & 1);
  const int j = blockIdx.x * blockDim.x + threadIdx.x + 2;
  const int i = blockIdx.y * blockDim.y + threadIdx.y + 2;
  if (j > g.jx - 2 || i > g.iy - 2) return;
  ps_column<R>(D, st, g.at2(j, i));
}

// Cross-point work after the boundary, per point: uvstagtouvx and
// temp_to_tvirt of boundary (:520-523), p (:348-352), the edits mkslice
// makes to the state (Main/mod_slice.F90:136-147: qx and tracer floors),
// then status_update (:1403-1443): tendencies, q clamps, tvirt, tetav, rho,
// qsat.  The surface pressure is extrapolated before, by k_end_ps.  Whole
// steps take k_end_point and k_end_winds instead unless they nudge spectrally.
//   kEndAll   the whole sequence with zero tendencies (mlc_step).  rho and
//             qsat of :348-352, and tvirt and tetav of the boundary, are
//             recomputed from the same inputs by status_update, so they are
//             computed once, after it.
//   kEndPre   up to mkslice: the state the physics reads.
//   kEndPost  status_update with the member's tendencies (Dom::tend).
constexpr int kEndAll = 0, kEndPre = 1, kEndPost = 2;
constexpr double kTracFloor = 1.0e-50;  // mkslice's tracer floor (Main/mod_slice.F90:141-147)
template <class R, int PH, int LV>
__global__ void k_end_cross(const Dom<R> *__restrict__ doms, int uvoff, int advoff, int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const Scal &c = D.c;
  const Stat<R> &sa = D.sa;
  const State<R> st = state_of(D, (D.clk->uv_role + uvoff) & 1, (D.clk->adv_role + advoff) & 1);
  const Pt q_ = point_at<LV>(wi, 1, 1);
  const int j = q_.j, i = q_.i;
  const int jx = g.jx, iy = g.iy, kz = g.kz;
  const int klo = q_.k, khi = min(kz, klo + LV - 1);
  if (j > jx - 1 || i > iy - 1 || klo > kz) return;
  const size_t ij = g.at2(j, i), PS = g.PS, F = g.field3(), S = (size_t)g.P;
  const bool inner = j >= 2 && j <= jx - 2 && i >= 2 && i <= iy - 2;
  const int ipp = c.ipptls;
#pragma unroll
  for (int k = klo; k <= khi; ++k) {
  const size_t o = ij + (size_t)(k - 1) * PS;
  if (PH != kEndPost && c.apply_bdy) {
    {
      const R *u = st.u, *v = st.v;
      R a;
      if (j == 1) a = R(0.5) * (u[o] + u[o + 1]);
      else if (j == jx - 1) a = R(0.5) * (u[o + 1] + u[o]);
      else a = interp4<R>(u[o + 1], u[o], u[o + 2], u[o - 1]);
      st.ux[o] = a;
      if (i == 1) a = R(0.5) * (v[o] + v[o + S]);
      else if (i == iy - 1) a = R(0.5) * (v[o + S] + v[o]);
      else a = interp4<R>(v[o + S], v[o], v[o + 2 * S], v[o - S]);
      st.vx[o] = a;
    }
  }
  // pressure (FP64 Exner reconstruction; FP32 for the FP32 field of a mixed member)
  if (PH != kEndPost) {
    if constexpr (sizeof(R) == sizeof(float)) st.p[o] = exner_to_pressure_f(df_f(DF(st.pai, F).ld(o)));
    else st.p[o] = (R)exner_to_pressure(st.pai[o]);
  }
  if (PH == kEndPre) {
    // the state at mkslice: tvirt and theta_v of the boundary (before the
    // floors), rho and qsat of :348-352, then mkslice's floors
    const R tk = st.t[o], pk = st.p[o];
    if (c.apply_bdy) {
      st.tvirt[o] = mul_r(tk, qfactor(st.qx, o, F, ipp));
      if constexpr (sizeof(R) == sizeof(float)) {
        const F2 t2{tk, D.wz[1][o]};
        DF(st.tetav, F).st(o, df_div(df_mul(t2, qfactor_df(st.qx, o, F, ipp)), DF(st.pai, F).ld(o)));
      } else {
        st.tetav[o] = div_d((double)st.tvirt[o], st.pai[o]);
      }
    }
    st.rho[o] = divide<R>(pk, mul_r(R(kRgas), tk));
    if constexpr (sizeof(R) == sizeof(float)) st.qsat[o] = pfwsat_f(tk, pk);
    else st.qsat[o] = (R)pfwsat_d((double)tk, (double)pk);
    if (inner) {
      for (int n = 0; n < g.nqx; ++n) {
        const size_t on = o + (size_t)n * F;
        if (below_pos<R>(st.qx[on], qx_check(n))) st.qx[on] = R(qx_zero(n));
      }
      for (int n = 0; n < g.ntr; ++n) {
        const size_t on = o + (size_t)n * F;
        if (below_pos<double>((double)st.trac[on], kTracFloor)) st.trac[on] = R(0);
      }
    }
    continue;
  }
  // status_update
  {
    const R *ten = PH == kEndPost ? D.tend : nullptr;
    if (inner) {
      if (ten) {
        // t, ux, vx += dtsec * tendency (a mixed member's t is a double-float)
        if constexpr (sizeof(R) == sizeof(float)) {
          const F2 t2 = df_add_f(F2{st.t[o], D.wz[1][o]}, c.dtsecf * ten[o]);
          st.t[o] = t2.hi;
          D.wz[1][o] = t2.lo;
          st.ux[o] = st.ux[o] + c.dtsecf * ten[o + F];
          st.vx[o] = st.vx[o] + c.dtsecf * ten[o + 2 * F];
        } else {
          st.t[o] = st.t[o] + c.dtsec * ten[o];
          st.ux[o] = st.ux[o] + c.dtsec * ten[o + F];
          st.vx[o] = st.vx[o] + c.dtsec * ten[o + 2 * F];
        }
      }
      const R dts = pick<R>(c.dtsec, c.dtsecf);
      // The whole step's mkslice floor and status_update clamp with zero
      // tendencies are one clamp: after the floor q >= check or q = zero, and
      // zero < check or zero = check, so the second clamp changes nothing (for
      // the tracers, the floor leaves no negative value)
      for (int n = 0; n < g.nqx; ++n) {
        const size_t on = o + (size_t)n * F;
        R q = st.qx[on];
        if (ten) q = q + dts * ten[o + (size_t)(3 + n) * F];
        if (below_pos<R>(q, qx_check(n))) q = R(qx_zero(n));
        st.qx[on] = q;
      }
      for (int n = 0; n < g.ntr; ++n) {
        const size_t on = o + (size_t)n * F;
        R q = st.trac[on];
        if (PH == kEndAll) {
          if (below_pos<double>((double)q, kTracFloor)) q = R(0);  // mkslice
        } else {
          if (ten) q = q + dts * ten[o + (size_t)(3 + g.nqx + n) * F];
          if (q < R(0)) q = R(0);
        }
        st.trac[on] = q;
      }
    }
    const R tk = st.t[o];
    const R qf = qfactor(st.qx, o, F, ipp);
    const R tv = mul_r(tk, qf);
    st.tvirt[o] = tv;
    const R pk = st.p[o];
    st.rho[o] = divide<R>(pk, mul_r(R(kRgas), tk));
    if constexpr (sizeof(R) == sizeof(float)) {
      // theta_v = tvirt/pai from the double-float t (Main/mod_moloch.F90:1403-1443):
      // where nothing relaxed t, t*qf/pai gives back theta_v to ~1e-14
      const F2 t2{tk, D.wz[1][o]};
      DF(st.tetav, F).st(o, df_div(df_mul(t2, qfactor_df(st.qx, o, F, ipp)), DF(st.pai, F).ld(o)));
      st.qsat[o] = pfwsat_f(tk, pk);
    } else {
      st.tetav[o] = div_d((double)tv, st.pai[o]);
      st.qsat[o] = (R)pfwsat_d((double)tk, (double)pk);
    }
  }
  }
}

// V elements at p in one access (4 to 16 bytes, aligned), and back where ok
template <class R, int V>
__device__ __forceinline__ void ldv(R (&x)[V], const R *p) {
  if constexpr (V == 1) {
    x[0] = *p;
  } else {
    static_assert(V * sizeof(R) == 16, "16-byte lanes");
    const uint4 w = *reinterpret_cast<const uint4 *>(p);
    memcpy(x, &w, 16);
  }
}
template <class R, int V>
__device__ __forceinline__ void stv(R *p, const R (&x)[V], const bool (&ok)[V], bool all) {
  if (V > 1 && all) {
    uint4 w;
    memcpy(&w, x, 16);
    *reinterpret_cast<uint4 *>(p) = w;
  } else {
#pragma unroll
    for (int q = 0; q < V; ++q)
      if (ok[q]) p[q] = x[q];
  }
}

// k_end_cross<kEndAll> of a mixed member in lanes of four columns (16-byte loads
// and stores, the same expressions): the end of steps that nudge spectrally.
// Bound by memory; with ps before it 211 us a step at 512x512x41 and 71 at
// 256x256x41, a point a thread 453 and 136.
template <class R, int LV>
__global__ void __launch_bounds__(128) k_end_cross_v4(const Dom<R> *__restrict__ doms, int uvoff, int advoff,
                                                      int tiles_j, const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  constexpr int V = 4;
  static_assert(sizeof(R) == sizeof(float), "FP32 fields");
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const Scal &c = D.c;
  const int jx = g.jx, iy = g.iy, kz = g.kz;
  const int e0 = ((int)wi.a * 32 + (int)threadIdx.x) * V, i = (int)wi.b * 4 + (int)threadIdx.y + 1;
  const int k0 = (int)wi.c * LV + 1;
  if (e0 + 1 > jx - 1 || i > iy - 1 || k0 > kz) return;
  const State<R> st = state_of(D, (D.clk->uv_role + uvoff) & 1, (D.clk->adv_role + advoff) & 1);
  const size_t F = g.field3();
  const unsigned P = (unsigned)g.P, PS = (unsigned)g.PS, ij = (unsigned)e0 + (unsigned)(i - 1) * P;
  const float *__restrict__ u = st.u + ij;
  const float *__restrict__ v = st.v + ij;
  const float *__restrict__ t_h = st.t + ij;
  const float *__restrict__ t_l = D.wz[1] + ij;
  const float *__restrict__ pai = reinterpret_cast<const float *>(st.pai) + ij;
  float *__restrict__ tet = reinterpret_cast<float *>(st.tetav) + ij;
  float *__restrict__ qx = st.qx + ij;
  float *__restrict__ trac = st.trac + ij;
  const int ipp = c.ipptls, nq = qfactor_species(ipp);
  bool has[V], inner[V], all = true, any_inner = false;
#pragma unroll
  for (int q = 0; q < V; ++q) {
    const int j = e0 + q + 1;
    has[q] = j <= jx - 1;
    inner[q] = j >= 2 && j <= jx - 2 && i >= 2 && i <= iy - 2;
    all = all && has[q];
    any_inner = any_inner || inner[q];
  }
  unsigned o = (unsigned)(k0 - 1) * PS;
  for (int k = k0; k < k0 + LV && k <= kz; ++k, o += PS) {
    if (c.apply_bdy) {
      // u at columns e0-1 .. e0+5 and v at rows i-1 .. i+2 (:1535-1566)
      float n[V + 3] = {}, m[V], a[V];
      ldv<R, V>(m, u + o);
      if (e0 >= 1) n[0] = (u + o)[-1];  // (o may be 0: no unsigned o - 1)
#pragma unroll
      for (int q = 0; q < V; ++q) n[1 + q] = m[q];
      if (e0 + 4 <= jx - 1) n[5] = u[o + 4];
      if (e0 + 5 <= jx - 1) n[6] = u[o + 5];
#pragma unroll
      for (int q = 0; q < V; ++q) {
        const int j = e0 + q + 1;
        a[q] = j == 1 || j == jx - 1 ? interp2<R>(n[q + 1], n[q + 2]) : interp4<R>(n[q + 2], n[q + 1], n[q + 3], n[q]);
      }
      stv<R, V>(st.ux + ij + o, a, has, all);
      float vs[V] = {}, vc[V], vn[V], vf[V] = {};
      ldv<R, V>(vc, v + o);
      ldv<R, V>(vn, v + o + P);
      const bool edge = i == 1 || i == iy - 1;
      if (!edge) {
        ldv<R, V>(vs, v + o - P);
        ldv<R, V>(vf, v + o + 2 * P);
      }
#pragma unroll
      for (int q = 0; q < V; ++q) a[q] = edge ? interp2<R>(vc[q], vn[q]) : interp4<R>(vn[q], vc[q], vf[q], vs[q]);
      stv<R, V>(st.vx + ij + o, a, has, all);
    }
    float ph[V], pl[V], pk[V], tk[V], tl[V], q[5][V];
    ldv<R, V>(ph, pai + o);
    ldv<R, V>(pl, pai + F + o);
    ldv<R, V>(tk, t_h + o);
    ldv<R, V>(tl, t_l + o);
#pragma unroll
    for (int n = 0; n < 5; ++n)
      if (n < nq) ldv<R, V>(q[n], qx + o + (size_t)n * F);
      else
#pragma unroll
        for (int e = 0; e < V; ++e) q[n][e] = 0.f;
    // the floors at inner points (see k_end_cross; in FP32 every tracer below
    // mkslice's is at most zero)
    if (any_inner) {
      auto floors = [&](float (&x)[V], float *p, double check, float zero) {
        bool ch = false;
#pragma unroll
        for (int e = 0; e < V; ++e)
          if (inner[e] && below_pos<R>(x[e], check)) {
            x[e] = zero;
            ch = true;
          }
        if (ch) stv<R, V>(p, x, has, all);
      };
#pragma unroll
      for (int n = 0; n < 5; ++n)
        if (n < nq) floors(q[n], qx + o + (size_t)n * F, qx_check(n), float(qx_zero(n)));
      for (int n = nq; n < g.nqx; ++n) {
        float x[V];
        ldv<R, V>(x, qx + o + (size_t)n * F);
        floors(x, qx + o + (size_t)n * F, qx_check(n), float(qx_zero(n)));
      }
      for (int n = 0; n < g.ntr; ++n) {
        float x[V];
        bool ch = false;
        ldv<R, V>(x, trac + o + (size_t)n * F);
#pragma unroll
        for (int e = 0; e < V; ++e)
          if (inner[e] && x[e] <= 0.f) {
            x[e] = 0.f;
            ch = true;
          }
        if (ch) stv<R, V>(trac + o + (size_t)n * F, x, has, all);
      }
    }
    float tv[V], rh[V], th[V], thl[V], qs[V];
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const float x[5] = {q[0][e], q[1][e], q[2][e], q[3][e], q[4][e]};
      pk[e] = exner_to_pressure_f(ph[e] + pl[e]);
      tv[e] = mul_r(tk[e], qfactor_of<R>(x, ipp));
      rh[e] = divide<R>(pk[e], mul_r(R(kRgas), tk[e]));
      // theta_v = tvirt/pai from the double-float t (Main/mod_moloch.F90:1403-1443)
      const F2 t2 = df_div(df_mul(F2{tk[e], tl[e]}, qfactor_df_of(x, ipp)), F2{ph[e], pl[e]});
      th[e] = t2.hi;
      thl[e] = t2.lo;
      qs[e] = pfwsat_f(tk[e], pk[e]);
    }
    stv<R, V>(st.p + ij + o, pk, has, all);
    stv<R, V>(st.tvirt + ij + o, tv, has, all);
    stv<R, V>(st.rho + ij + o, rh, has, all);
    stv<R, V>(tet + o, th, has, all);
    stv<R, V>(tet + F + o, thl, has, all);
    stv<R, V>(st.qsat + ij + o, qs, has, all);
  }
}

// A whole step's pointwise end in one pass (steps that nudge spectrally take
// k_end_relax and k_end_cross): virtual temperature and temperature of
// dynamical_core :1121-1123, motopnudge (Main/mod_bdycod.F90:4049-4083) and
// morelax on every field (boundary, Main/mod_moloch.F90:478-497), p
// (:348-352), mkslice's floors and status_update with zero tendencies
// (:1403-1443), rho and qsat; the virtual temperatures that ps is extrapolated
// from go to the scratch plane wz[0].
//
// Two launches share the points.  FRAME: the ring and the relaxation zone
// (Scal::frame points deep), a point a thread.  Else the points inside it,
// lanes of 16 bytes of a row (two FP64 or four FP32 columns), where a level is
// nudged as a whole or not at all and no lane leaves the common path; with the
// zone's code in the same warps every row of a 128-column domain ran it four
// columns at a time (1000 us a step for 32 members of 128x128x30; 483 now, the
// passes before it 819).  Seven and ten blocks an SM: measured best of three to
// twelve, by up to a quarter.
// Bound by the FP64 pipe or, mixed, by memory: 56 bytes a point at five
// species, where the passes it replaces moved 140 (t and its low part,
// theta_v, Exner and the species went through memory between them).
// Mixed: where nothing changed t or the species of its factor and t is finite,
// theta_v is what it was and is left alone.  FP64 forms t*qf/pai everywhere, as the split step
// does (the two are bit for bit equal).
// us a step, this pass and k_end_winds against k_end_relax, k_end_cross and
// k_end_uvstag: mixed 512x512x41 258 against 546, 12 uneven domains 325 against
// 619; FP64 512x512x41 1765 (with k_end_uvx and k_end_uvstag) against 2180.
template <class R, int LV, bool FRAME>
__global__ void __launch_bounds__(128, FRAME ? 10 : 7) k_end_point(const Dom<R> *__restrict__ doms, int uvoff, int advoff,
                                                   int tiles_j, const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  constexpr int V = FRAME ? 1 : 16 / (int)sizeof(R);
  constexpr bool mixed = sizeof(R) == sizeof(float);
  const WorkItem wi = FRAME ? WorkItem{(int16_t)blockIdx.z, 0, 0, (int16_t)blockIdx.y} : work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const Scal &c = D.c;
  const int jx = g.jx, iy = g.iy, kz = g.kz, fr = c.frame;
  const int k0 = (int)wi.c * LV + 1;
  if (k0 > kz) return;
  int e0, i;  // 0-based first column, row
  if constexpr (FRAME) {
    // the south and north rows of the frame, then its columns between them
    const int nx = jx - 1, ny = iy - 1;
    const int s = min(fr, ny), n = min(fr, ny - s), w = min(fr, nx), we = w + min(fr, nx - w);
    int e = (int)(blockIdx.x * 128u + threadIdx.x);
    if (e < (s + n) * nx) {
      const int r = e / nx;
      e0 = e - r * nx;
      i = r < s ? r + 1 : ny - (r - s);
    } else {
      e -= (s + n) * nx;
      const int r = e / we, q = e - r * we;
      if (r >= ny - s - n) return;
      i = s + 1 + r;
      e0 = q < w ? q : nx - we + q;
    }
  } else {
    e0 = ((int)wi.a * 32 + (int)(threadIdx.x & 31u)) * V;
    i = (int)wi.b * 4 + (int)(threadIdx.x >> 5) + 1;
    if (e0 + V - 1 < fr || e0 > jx - 2 - fr || i <= fr || i > iy - 1 - fr) return;
  }
  const Stat<R> &sa = D.sa;
  const Bdy<R> &bd = D.bd;
  const Clock *clk = D.clk;
  const State<R> st = state_of(D, (clk->uv_role + uvoff) & 1, (clk->adv_role + advoff) & 1);
  const size_t F = g.field3();
  const unsigned PS = (unsigned)g.PS, ij = (unsigned)e0 + (unsigned)(i - 1) * (unsigned)g.P;
  const R *__restrict__ th_p = reinterpret_cast<const R *>(st.tetav);
  const R *__restrict__ pa_p = reinterpret_cast<const R *>(st.pai);
  R *__restrict__ qx = st.qx;
  const bool bdy = c.apply_bdy != 0;
  // the lane's own columns, and in the frame whether its point is inside the
  // ring and its zone as a cross, u and v point (0: not in the zone, -2: no
  // point that the boundary changes)
  bool has[V], all = true;
#pragma unroll
  for (int e = 0; e < V; ++e) {
    has[e] = FRAME || (e0 + e >= fr && e0 + e <= jx - 2 - fr);
    all = all && has[e];
  }
  bool inner = true;
  int ibc = 0, ibu = 0, ibv = 0;
  if constexpr (FRAME) {
    const int j = e0 + 1;
    inner = j >= 2 && j <= jx - 2 && i >= 2 && i <= iy - 2;
    ibc = bdy && inner ? sa.ibnd_cr[ij] : -2;
    ibu = bdy && j >= 2 && i >= 2 && i <= iy - 2 ? sa.ibnd_ud[ij] : -2;
    ibv = bdy && j >= 2 && i >= 2 && j <= jx - 2 ? sa.ibnd_vd[ij] : -2;
  }
  const bool zone = ibc > 0 || ibu > 0 || ibv > 0;
  const int ipp = c.ipptls, nq = qfactor_species(ipp), nztop = bdy && c.top_nudge ? c.nztop : 0;
  // the boundary clock has moved by dtsec (Main/mod_bdycod.F90:2653)
  double x0 = 0.0, x1 = 0.0, cx0 = 0.0, cx1 = 0.0;
  if (zone || k0 <= nztop) {
    const double xb = clk->xbctime + c.dtsec;
    x1 = (xb + c.dt) * c.rtb;
    x0 = 1.0 - x1;
    if (FRAME && g.ntr) {
      cx1 = (xb + c.dt) / c.dtbdys;
      cx0 = 1.0 - cx1;
    }
  }
  const R rx0 = R(x0), rx1 = R(x1);
  constexpr double trtau = 1.0 / (2.0 * 3600.0), wrtau = 1.0 / (3600.0 / 4.0);
#pragma unroll 1
  for (int k = k0; k < k0 + LV && k <= kz; ++k) {
    const unsigned o = ij + (unsigned)(k - 1) * PS;
    R th[V], pa[V], thl[V], pal[V], q[5][V];
    ldv<R, V>(th, th_p + o);
    ldv<R, V>(pa, pa_p + o);
    if constexpr (mixed) {
      ldv<R, V>(thl, th_p + F + o);
      ldv<R, V>(pal, pa_p + F + o);
    }
#pragma unroll
    for (int n = 0; n < 5; ++n)
      if (n < nq) ldv<R, V>(q[n], qx + o + (size_t)n * F);
      else
#pragma unroll
        for (int e = 0; e < V; ++e) q[n][e] = R(0);
    auto species = [&](int e, R (&x)[5]) {
#pragma unroll
      for (int n = 0; n < 5; ++n) x[n] = q[n][e];
    };
    // ---- tvirt and t (t of the ring is the boundary's) ----
    R t[V], tl[V], tv[V], qf[V];  // FP64: t, theta_v*pai, the factor; mixed: t and its low part, theta_v*pai
    bool chg[V];                  // theta_v is formed anew
#pragma unroll
    for (int e = 0; e < V; ++e) {
      R x[5];
      species(e, x);
      chg[e] = !inner;
      if constexpr (mixed) {
        const F2 v2 = df_mul(F2{th[e], thl[e]}, F2{pa[e], pal[e]});
        const F2 t2 = inner ? df_div(v2, qfactor_df_of(x, ipp)) : F2{st.t[o], bdy ? D.wz[1][o] : 0.f};
        t[e] = t2.hi;
        tl[e] = t2.lo;
        tv[e] = df_f(v2);
        // a species that is not finite reaches theta_v and tvirt through t
        chg[e] = chg[e] || !isfinite(t2.hi);
      } else {
        tv[e] = mul_r(th[e], pa[e]);
        qf[e] = qfactor_of<R>(x, ipp);
        t[e] = inner ? divide<R>(tv[e], qf[e]) : st.t[o];
      }
    }
    // ---- motopnudge and morelax ----
    const bool nud = k <= nztop;
    R xfn = R(0);
    if (nud) {
      if constexpr (mixed) xfn = mul_r(sa.tnudge_r[k - 1], float(trtau * c.dtsec));
      else xfn = sa.tnudge[k - 1] * trtau * c.dtsec;
    }
    if (k == 2 && bdy && c.top_nudge && inner) {  // w sponge, before the level's relaxation
      const R xf = R(wrtau * c.dtsec);
      R w2[V];
      ldv<R, V>(w2, st.w + o);
#pragma unroll
      for (int e = 0; e < V; ++e) w2[e] = bdy_relax_to<R>(w2[e], xf, R(0) * w2[e]);
      stv<R, V>(st.w + o, w2, has, all);
    }
    if (nud || zone) {
      const R *hefc = sa.hefc_r + (size_t)(k - 1) * c.nspgx - 1;  // hefc[zone]
      // nudged, then relaxed in the zone
      auto wind = [&](R *f, const R *const *b, int ib) {
        if (ib == -2 || !(nud || ib > 0)) return;
        R x[V], b0[V], b1[V];
        ldv<R, V>(x, f + o);
        ldv<R, V>(b0, b[0] + o);
        ldv<R, V>(b1, b[1] + o);
#pragma unroll
        for (int e = 0; e < V; ++e) {
          const R ext = bdy_blend<R>(rx0, rx1, b0[e], b1[e]);
          if (nud) x[e] = bdy_relax_to<R>(x[e], xfn, ext);
          if (FRAME && ib > 0) x[e] = bdy_relax_to<R>(x[e], hefc[ib], ext);
        }
        stv<R, V>(f + o, x, has, all);
      };
      wind(st.u, bd.dub, ibu);
      wind(st.v, bd.dvb, ibv);
      if (ibc != -2 && (nud || ibc > 0)) {
        const R *b0p = reinterpret_cast<const R *>(bd.xtb[0]), *b1p = reinterpret_cast<const R *>(bd.xtb[1]);
        R b0[V], b1[V], b0l[V], b1l[V];
        ldv<R, V>(b0, b0p + o);
        ldv<R, V>(b1, b1p + o);
        if constexpr (mixed) {
          ldv<R, V>(b0l, b0p + F + o);
          ldv<R, V>(b1l, b1p + F + o);
        }
#pragma unroll
        for (int e = 0; e < V; ++e) {
          chg[e] = true;
          if constexpr (mixed) {
            // (1-x)*t + x*b as t + x*(b - t) on the double-float t
            const F2 a{b0[e], b0l[e]};
            const F2 bt = df_add_f(a, mul_r(float(x1), df_diff(F2{b1[e], b1l[e]}, a)));
            F2 t2{t[e], tl[e]};
            if (nud) t2 = df_add_f(t2, mul_r(xfn, df_diff(bt, t2)));
            if (FRAME && ibc > 0) t2 = df_add_f(t2, mul_r(hefc[ibc], df_diff(bt, t2)));
            t[e] = t2.hi;
            tl[e] = t2.lo;
          } else {
            const double bt = bdy_blend<double>(x0, x1, b0[e], b1[e]);
            if (nud) t[e] = bdy_relax_to<R>(t[e], xfn, bt);
            if (FRAME && ibc > 0) t[e] = bdy_relax_to<R>(t[e], hefc[ibc], bt);
          }
        }
      }
      if constexpr (FRAME) {
        if (ibc > 0) {
          const R xf = hefc[ibc];
          auto blend = [&](const R *const *b, size_t at) { return bdy_blend<R>(rx0, rx1, b[0][at], b[1][at]); };
          if constexpr (mixed) {
            const DF b0(bd.xpaib[0], F), b1(bd.xpaib[1], F);
            const F2 pp{pa[0], pal[0]}, a = b0.ld(o);
            const F2 pn = df_add_f(pp, mul_r(xf, fmaf(float(x1), df_diff(b1.ld(o), a), df_diff(a, pp))));
            DF(st.pai, F).st(o, pn);
            pa[0] = pn.hi;
            pal[0] = pn.lo;
          } else {
            pa[0] = bdy_relax_to<double>(pa[0], xf, bdy_blend<double>(x0, x1, bd.xpaib[0][o], bd.xpaib[1][o]));
            st.pai[o] = pa[0];
          }
          q[0][0] = bdy_relax_to<R>(q[0][0], xf, blend(bd.xqb, o));
          qx[o] = q[0][0];
          {
            // morelax_fraction with frac = 0 (:3962-3993)
            const R f = st.w[o];
            st.w[o] = bdy_relax_to<R>(f, xf, f * R(0));
          }
          if (ipp > 0 && c.present_qc) {
            q[1][0] = bdy_relax_to<R>(q[1][0], xf, blend(bd.xlb, o));
            qx[o + F] = q[1][0];
          }
          if (ipp > 1 && c.present_qi) {
            q[2][0] = bdy_relax_to<R>(q[2][0], xf, blend(bd.xib, o));
            qx[o + 2 * F] = q[2][0];
          }
          for (int n = 0; n < g.ntr; ++n) {
            const size_t on = o + (size_t)n * F;
            st.trac[on] = bdy_relax_to<R>(st.trac[on], sa.fcx_r[ibc - 1],
                                          bdy_blend<R>(R(cx0), R(cx1), bd.chib[0][on], bd.chib[1][on]));
          }
          if constexpr (!mixed) {
            R x[5];
            species(0, x);
            qf[0] = qfactor_of<R>(x, ipp);
          }
        }
      }
    }
    // ---- the virtual temperatures of ps, before the clamps ----
    if (k >= kz - 1) {
      R x2[V];
#pragma unroll
      for (int e = 0; e < V; ++e) {
        x2[e] = tv[e];
        if constexpr (mixed) {
          if (bdy && chg[e]) {
            R x[5];
            species(e, x);
            x2[e] = mul_r(t[e], qfactor_of<R>(x, ipp));
          }
        } else {
          if (bdy) x2[e] = mul_r(t[e], qf[e]);
        }
      }
      stv<R, V>(D.wz[0] + o, x2, has, all);
    }
    // ---- mkslice's floors, then status_update's clamps with zero tendencies,
    // one clamp (see k_end_cross); the ring keeps its values ----
    if (inner) {
#pragma unroll
      for (int n = 0; n < 5; ++n) {
        if (n >= nq) break;
        bool ch = false;
#pragma unroll
        for (int e = 0; e < V; ++e)
          // (a value that is its floor already changes nothing)
          if (has[e] && below_pos<R>(q[n][e], qx_check(n)) && bits_differ(q[n][e], R(qx_zero(n)))) {
            q[n][e] = R(qx_zero(n));
            chg[e] = ch = true;
          }
        if (ch) stv<R, V>(qx + o + (size_t)n * F, q[n], has, all);
      }
      for (int n = nq; n < g.nqx; ++n) {
        R x[V];
        bool ch = false;
        ldv<R, V>(x, qx + o + (size_t)n * F);
#pragma unroll
        for (int e = 0; e < V; ++e)
          if (has[e] && below_pos<R>(x[e], qx_check(n)) && bits_differ(x[e], R(qx_zero(n)))) {
            x[e] = R(qx_zero(n));
            ch = true;
          }
        if (ch) stv<R, V>(qx + o + (size_t)n * F, x, has, all);
      }
      for (int n = 0; n < g.ntr; ++n) {
        R x[V];
        bool ch = false;
        ldv<R, V>(x, st.trac + o + (size_t)n * F);
#pragma unroll
        for (int e = 0; e < V; ++e) {
          // FP32 holds nothing between zero and the floor
          const bool low = mixed ? x[e] <= R(0) : below_pos<double>((double)x[e], kTracFloor);
          if (has[e] && low && bits_differ(x[e], R(0))) {
            x[e] = R(0);
            ch = true;
          }
        }
        if (ch) stv<R, V>(st.trac + o + (size_t)n * F, x, has, all);
      }
    }
    // ---- diagnostics and theta_v ----
    R pp[V], rh[V], qs[V], thn[V], thn_l[V];
    bool any = false;
#pragma unroll
    for (int e = 0; e < V; ++e) {
      R x[5];
      species(e, x);
      any = any || chg[e];
      if constexpr (mixed) {
        pp[e] = exner_to_pressure_f(pa[e] + pal[e]);
        thn[e] = th[e];
        thn_l[e] = thl[e];
        if (chg[e]) {
          const F2 v2 = df_mul(F2{t[e], tl[e]}, qfactor_df_of(x, ipp));
          const F2 t2 = df_div(v2, F2{pa[e], pal[e]});
          tv[e] = mul_r(t[e], qfactor_of<R>(x, ipp));
          thn[e] = t2.hi;
          thn_l[e] = t2.lo;
        }
        qs[e] = pfwsat_f(t[e], pp[e]);
      } else {
        pp[e] = exner_to_pressure(pa[e]);
        if (chg[e]) qf[e] = qfactor_of<R>(x, ipp);
        tv[e] = mul_r(t[e], qf[e]);
        thn[e] = div_d(tv[e], pa[e]);
        qs[e] = pfwsat_d(t[e], pp[e]);
      }
      rh[e] = divide<R>(pp[e], mul_r(R(kRgas), t[e]));
    }
    if (inner) stv<R, V>(st.t + o, t, has, all);
    stv<R, V>(st.tvirt + o, tv, has, all);
    stv<R, V>(st.p + o, pp, has, all);
    stv<R, V>(st.rho + o, rh, has, all);
    stv<R, V>(st.qsat + o, qs, has, all);
    if (!mixed || any) {
      R *th_o = reinterpret_cast<R *>(st.tetav);
      stv<R, V>(th_o + o, thn, has, all);
      if constexpr (mixed) stv<R, V>(th_o + F + o, thn_l, has, all);
    }
  }
}

// A whole step's winds at its end: ux, vx from the relaxed u, v (boundary
// :520-523, uvstagtouvx :1535-1566; the advected ux, vx with the boundary off)
// and u, v from them (uvxtouvstag, status_update :1440).  The new winds go to
// the other half of their pairs, because the stencils of other tiles still
// read the old ones.  A warp marches `rows` rows along i, holding four rows of
// v and of vx in registers; a lane holds four columns, whose neighbours along
// j come by shuffles, so a warp's 128 columns write the middle 120.  Each
// field is read and written once, a row ahead of its use.  Bound by memory: 67
// us at 512x512x41 (24 bytes a point: 38), 120 as two point passes.  FP64
// members keep the two passes (k_end_uvx, k_end_uvstag): their arithmetic is
// the bound there, and this form does a fifth more of it for its halo (503
// against 383 us).
template <class R>
__global__ void __launch_bounds__(32 * kWindWarps) k_end_winds(const Dom<R> *__restrict__ doms, int uvoff,
                                                               int advoff, int rows, int tiles_j,
                                                               const WorkItem *__restrict__ wl) {
  grid_begin();
  constexpr int V = 4;
  static_assert(sizeof(R) == sizeof(float), "FP32 fields");
  static_assert(kWindCols == 32 * V - 8, "a lane either side is halo");
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const int jx = g.jx, iy = g.iy, k = (int)wi.c + 1;
  if (k > g.kz) return;
  const int lane = (int)threadIdx.x & 31;
  const int i0 = ((int)wi.b * kWindWarps + ((int)threadIdx.x >> 5)) * rows + 1;
  if (i0 > iy) return;  // (a warp)
  const int i1 = min(i0 + rows - 1, iy);
  const int e0 = (int)wi.a * kWindCols - V + V * lane;
  const bool inrow = e0 >= 0 && e0 + V <= g.P, wr = inrow && lane >= 1 && lane <= 30 && e0 < jx;
  const bool ends = e0 <= 1 || e0 + V >= jx - 1;  // the lane holds columns near the domain's first or last
  const bool bdy = D.c.apply_bdy != 0;
  const int uv = (D.clk->uv_role + uvoff) & 1, adv = (D.clk->adv_role + advoff) & 1;
  const unsigned ko = (unsigned)(k - 1) * (unsigned)g.PS, P = (unsigned)g.P;
  const R *__restrict__ u_in = D.u[uv] + ko;
  const R *__restrict__ v_in = D.v[uv] + ko;
  R *__restrict__ u_out = D.u[uv ^ 1] + ko;
  R *__restrict__ v_out = D.v[uv ^ 1] + ko;
  R *ux = D.ux[adv] + ko;
  R *vx = D.vx[adv] + ko;
  auto load = [&](R (&x)[V], const R *p, int r, int rmax) {
    if (inrow && r >= 1 && r <= rmax) {
      ldv<R, V>(x, p + (unsigned)e0 + (unsigned)(r - 1) * P);
    } else {
#pragma unroll
      for (int q = 0; q < V; ++q) x[q] = R(0);
    }
  };
  // (the columns past a field's last lie in the row's padding)
  auto store = [&](R *p, int r, const R (&x)[V]) {
    if (!wr) return;
    *reinterpret_cast<float4 *>(p + (unsigned)e0 + (unsigned)(r - 1) * P) = make_float4(x[0], x[1], x[2], x[3]);
  };
  const unsigned full = 0xffffffffu;
  auto pick4 = [](const R (&n)[V + 3], int lo, int q) {  // n[lo + q], q in 0 .. 3
    return q == 0 ? n[lo] : q == 1 ? n[lo + 1] : q == 2 ? n[lo + 2] : n[lo + 3];
  };
  // rows r-1 .. r+2 of v, and r-3 .. r-1 of vx
  R va[V], vb[V], vc[V], vd[V], xa[V], xb[V], xc[V];
  // the next rows of v and u, loaded a row ahead
  R vn[V], un[V];
  load(va, v_in, i0 - 3, iy);
  load(vb, v_in, i0 - 2, iy);
  load(vc, v_in, i0 - 1, iy);
  load(vn, v_in, i0, iy);
  load(un, u_in, i0, iy - 1);
#pragma unroll
  for (int q = 0; q < V; ++q) xa[q] = xb[q] = xc[q] = R(0);
  for (int r = i0 - 2; r <= i1 + 1; ++r) {
#pragma unroll
    for (int q = 0; q < V; ++q) vd[q] = vn[q];
    load(vn, v_in, r + 3, r < i1 + 1 ? iy : 0);
    // vx of row r
    R x[V];
    if (!bdy) {
      load(x, vx, r, iy - 1);
    } else {
      if (r == 1 || r == iy - 1) {  // (a warp)
#pragma unroll
        for (int q = 0; q < V; ++q) x[q] = interp2<R>(vb[q], vc[q]);
      } else {
#pragma unroll
        for (int q = 0; q < V; ++q) x[q] = interp4<R>(vc[q], vb[q], vd[q], va[q]);
      }
      if (r >= i0 && r <= i1 && r <= iy - 1) store(vx, r, x);
    }
    // v of row r-1, from vx of rows r-3 .. r
    const int ro = r - 1;
    if (ro >= i0) {
      R y[V];
      if (ro < 2 || ro > iy - 1) {
#pragma unroll
        for (int q = 0; q < V; ++q) y[q] = va[q];
      } else if (ro == 2 || ro == iy - 1) {
#pragma unroll
        for (int q = 0; q < V; ++q) y[q] = interp2<R>(xb[q], xc[q]);
      } else {
#pragma unroll
        for (int q = 0; q < V; ++q) y[q] = interp4<R>(xc[q], xb[q], x[q], xa[q]);
      }
      if (ends) {  // v keeps its values at the first and last column
#pragma unroll
        for (int q = 0; q < V; ++q)
          if (e0 + q + 1 < 2 || e0 + q + 1 > jx - 2) y[q] = va[q];
      }
      store(v_out, ro, y);
    }
    // ux and u of row r
    if (r >= i0 && r <= i1 && r <= iy - 1) {
      R u[V], a[V], y[V];
#pragma unroll
      for (int q = 0; q < V; ++q) u[q] = un[q];
      load(un, u_in, r + 1, r < i1 ? iy - 1 : 0);
      if (!bdy) {
        load(a, ux, r, iy - 1);
      } else {
        const R uw = __shfl_up_sync(full, u[V - 1], 1);
        const R ue = __shfl_down_sync(full, u[0], 1), uf = __shfl_down_sync(full, u[1], 1);
        const R n[V + 3] = {uw, u[0], u[1], u[2], u[3], ue, uf};  // columns -1 .. V+1
#pragma unroll
        for (int q = 0; q < V; ++q) a[q] = interp4<R>(n[q + 2], n[q + 1], n[q + 3], n[q]);
        if (ends) {  // columns 1 and jx-1, one a lane at most
          const R x = e0 == 0 ? interp2<R>(n[1], n[2]) : interp2<R>(pick4(n, 1, jx - 2 - e0), pick4(n, 2, jx - 2 - e0));
#pragma unroll
          for (int q = 0; q < V; ++q)
            if (e0 + q + 1 == 1 || e0 + q + 1 == jx - 1) a[q] = x;
        }
        store(ux, r, a);
      }
      const R x1 = __shfl_up_sync(full, a[V - 1], 1), x2 = __shfl_up_sync(full, a[V - 2], 1);
      const R xe = __shfl_down_sync(full, a[0], 1);
      const R n[V + 3] = {x2, x1, a[0], a[1], a[2], a[3], xe};  // columns -2 .. V
      if (r < 2 || r > iy - 2) {
#pragma unroll
        for (int q = 0; q < V; ++q) y[q] = u[q];
      } else {
#pragma unroll
        for (int q = 0; q < V; ++q) y[q] = interp4<R>(n[q + 2], n[q + 1], n[q + 3], n[q]);
        if (ends) {  // columns 2 and jx-1
          const R x = e0 == 0 ? interp2<R>(n[2], n[3]) : interp2<R>(pick4(n, 1, jx - 2 - e0), pick4(n, 2, jx - 2 - e0));
#pragma unroll
          for (int q = 0; q < V; ++q) {
            const int j = e0 + q + 1;
            if (j == 2 || j == jx - 1) y[q] = x;
            else if (j < 2 || j > jx - 1) y[q] = u[q];
          }
        }
      }
      store(u_out, r, y);
    }
#pragma unroll
    for (int q = 0; q < V; ++q) {
      va[q] = vb[q]; vb[q] = vc[q]; vc[q] = vd[q];
      xa[q] = xb[q]; xb[q] = xc[q]; xc[q] = x[q];
    }
  }
}

// ux, vx from the relaxed u, v (boundary :520-523, uvstagtouvx :1535-1566)
template <class R, int LV>
__global__ void k_end_uvx(const Dom<R> *__restrict__ doms, int uvoff, int advoff, int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active || !D.c.apply_bdy) return;
  const Geom g = D.g;
  const int uv = (D.clk->uv_role + uvoff) & 1, adv = (D.clk->adv_role + advoff) & 1;
  const R *__restrict__ u = D.u[uv];
  const R *__restrict__ v = D.v[uv];
  R *__restrict__ ux = D.ux[adv];
  R *__restrict__ vx = D.vx[adv];
  const Pt q = point_at<LV>(wi, 1, 1);
  const int j = q.j, i = q.i, jx = g.jx, iy = g.iy;
  if (j > jx - 1 || i > iy - 1 || q.k > g.kz) return;
  const size_t ij = g.at2(j, i), S = (size_t)g.P;
#pragma unroll
  for (int k = q.k; k < q.k + LV && k <= g.kz; ++k) {
    const size_t o = ij + (size_t)(k - 1) * g.PS;
    ux[o] = j == 1 || j == jx - 1 ? interp2<R>(u[o], u[o + 1]) : interp4<R>(u[o + 1], u[o], u[o + 2], u[o - 1]);
    vx[o] = i == 1 || i == iy - 1 ? interp2<R>(v[o], v[o + S])
                                  : interp4<R>(v[o + S], v[o], v[o + 2 * S], v[o - S]);
  }
}

// uvxtouvstag at the end of status_update (:1440)
template <class R, int LV>
__global__ void k_end_uvstag(const Dom<R> *__restrict__ doms, int uvoff, int advoff, int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const int uv = (D.clk->uv_role + uvoff) & 1, adv = (D.clk->adv_role + advoff) & 1;
  const R *__restrict__ ux = D.ux[adv];
  const R *__restrict__ vx = D.vx[adv];
  R *__restrict__ u = D.u[uv];
  R *__restrict__ v = D.v[uv];
  const Pt q_ = point_at<LV>(wi, 1, 1);
  const int j = q_.j, k0 = q_.k;
  if (k0 > g.kz) return;
  const int i = q_.i;
  const int jx = g.jx, iy = g.iy;
  if (j > jx || i > iy) return;
  const size_t ij = g.at2(j, i), PS = g.PS, S = (size_t)g.P;
  const bool do_u = (j >= 2 && j <= jx - 1 && i >= 2 && i <= iy - 2);
  const bool do_v = (j >= 2 && j <= jx - 2 && i >= 2 && i <= iy - 1);
  if (!do_u && !do_v) return;
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
  }
}

// Mass budget (Main/mod_massck.F90:77-170) and ps extrema.  The member's
// blocks sum their rows in a fixed order and write seven partials each; the
// last block to finish adds them in a fixed order, so the result does not
// depend on scheduling and a domain gives the same bits alone or in a batch.
constexpr int kRedThreads = 256;
constexpr int kRedWarps = kRedThreads / 32;
constexpr int kNPart = 7;  // dry, dryadv, qmass, qadv, ps max, ps min, non-finite flag

// dz of the member's field type (the FP32 copy for a mixed member)
template <class R>
__device__ __forceinline__ const R *pick_dz(const Stat<R> &sa) {
  if constexpr (sizeof(R) == sizeof(float)) return sa.dz_r;
  else return sa.dz;
}

// A block's sums: every warp's by shuffles, then the first warp adds the
// warps'.  The result is thread 0's.
struct RedSum {
  double dry, dadv, qm, qadv;
  long long pmax, pmin;  // keys of ps
  int bad;
};
// a double's pattern ordered like its value, as a signed integer (its own
// inverse on the patterns): maxima on the integer pipe
__device__ __forceinline__ long long order_key(long long b) { return b ^ ((b >> 63) & 0x7fffffffffffffffLL); }
__device__ __forceinline__ RedSum red_zero() {
  return {0, 0, 0, 0, order_key(__double_as_longlong(-INFINITY)), order_key(__double_as_longlong(INFINITY)), 0};
}
__device__ __forceinline__ void red_step(RedSum &a, int off, bool flux) {
  const unsigned full = 0xffffffffu;
  a.dry += __shfl_down_sync(full, a.dry, off);
  a.qm += __shfl_down_sync(full, a.qm, off);
  if (flux) {
    a.dadv += __shfl_down_sync(full, a.dadv, off);
    a.qadv += __shfl_down_sync(full, a.qadv, off);
  }
  a.pmax = max(a.pmax, __shfl_down_sync(full, a.pmax, off));
  a.pmin = min(a.pmin, __shfl_down_sync(full, a.pmin, off));
  a.bad |= __shfl_down_sync(full, a.bad, off);
}
// flux: whether the warp holds lateral fluxes
__device__ __forceinline__ RedSum red_block(RedSum a, bool flux, RedSum *sh) {
  const int warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31;
  for (int off = 16; off > 0; off >>= 1) red_step(a, off, flux);
  if (lane == 0) sh[warp] = a;
  __syncthreads();
  if (warp == 0) {
    a = sh[lane < kRedWarps ? lane : 0];
    for (int off = kRedWarps / 2; off > 0; off >>= 1) red_step(a, off, true);
  }
  return a;
}

// The boundary clock, the step count and the buffer roles of the next step.
__device__ __forceinline__ void advance_clock(const Scal &c, Clock *clk, int uvoff, int advoff) {
  if (c.apply_bdy) clk->xbctime = clk->xbctime + c.dtsec;
  if (c.apply_bdy && c.spectral) clk->tspectral = clk->tspectral + c.dtsec;
  clk->step = clk->step + 1;
  clk->uv_role = (clk->uv_role + uvoff) & 1;
  clk->adv_role = (clk->adv_role + advoff) & 1;
}
// The same after a budget that ran beside the winds (which read the roles): a
// member a thread.
template <class R>
__global__ void k_end_advance(const Dom<R> *__restrict__ doms, int nmem, int uvoff, int advoff) {
  grid_begin();
  const int m = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (m >= nmem || !doms[m].active) return;
  advance_clock(doms[m].c, doms[m].clk, uvoff, advoff);
}

// Partial sums of the mass budget and the ps extrema of one member, per block.
// Interior rows go to warps, lanes along the row in 16-byte vectors (every row
// starts on 128 bytes); the species of a point are summed before they are
// weighted by its dry mass, and dx^2 and dt*dx are applied to the sums.  FP32
// members: dz is the double-float {dz_r, dz_lo}, dz*rho, the species' sum and
// its share are double-floats, and so are the running sums (about 1e-14
// relative against the FP64 sums of the same FP32 state).  The lateral fluxes
// and ps are grid-stride loops over their own items.  form_ps: ps is
// extrapolated here, from the virtual temperatures k_end_point left in wz[0].
// (Row pieces a warp instead of flat vectors with two integer divisions each,
// the species summed first, a block instead of a warp adding the partials, and
// ps formed here: 110 us a step at 512x512x41 mixed, 182 FP64, against 113 and
// 230 without ps; 20 against 25 and 28 at 64x64x30.)
template <class R>
__global__ void __launch_bounds__(kRedThreads) k_reduce_partial(const Dom<R> *__restrict__ doms,
                                                                int uvoff, int advoff, int form_ps, int advance) {
  grid_begin();
  __shared__ RedSum sh[kRedWarps];
  __shared__ bool last;
  const Dom<R> &D = doms[blockIdx.y];
  if (!D.active) return;
  const int nb = D.red_blocks;
  if ((int)blockIdx.x >= nb) return;
  const Geom g = D.g;
  const Scal &c = D.c;
  const Stat<R> &sa = D.sa;
  const State<R> st = state_of(D, (D.clk->uv_role + uvoff) & 1, (D.clk->adv_role + advoff) & 1);
  const int jx = g.jx, iy = g.iy, kz = g.kz, nqx = g.nqx;
  const size_t F = g.field3();
  const int lane = (int)threadIdx.x & 31;
  const int gt = (int)(blockIdx.x * kRedThreads + threadIdx.x), gs = nb * kRedThreads;
  RedSum a = red_zero();
  bool flux = false;
  if (c.debug_level > 0) {
    constexpr int V = 16 / (int)sizeof(R);
    const R *__restrict__ dzp = pick_dz<R>(sa);
    const R *__restrict__ rho = st.rho;
    const R *__restrict__ qx = st.qx;
    F2 dry2{0.f, 0.f}, qm2{0.f, 0.f};
    // a warp's items: pieces of 32*V columns of the interior rows, in order;
    // two items' loads in flight
    const int ni = iy - 3, np = (jx - 2 + 32 * V - 1) / (32 * V), items = ni * kz * np;
    const int nw = nb * kRedWarps, per = (items + nw - 1) / nw;
    const int t0 = (gt >> 5) * per, t1 = min(items, t0 + per);
#pragma unroll 2
    for (int it = t0; it < t1; ++it) {
      const int r = it / np, kk = r / ni, ii = r - kk * ni + 1;  // 0-based level and row
      const int e = (it - r * np) * 32 * V + lane * V;
      if (e >= jx - 2) continue;
      const size_t o = (size_t)kk * g.PS + (size_t)ii * g.P + e;
      R dz[V], rh[V], q[5][V];
      ldv<R, V>(dz, dzp + o);
      ldv<R, V>(rh, rho + o);
#pragma unroll
      for (int n = 0; n < 5; ++n)
        if (n < nqx) ldv<R, V>(q[n], qx + o + (size_t)n * F);
      if constexpr (sizeof(R) == sizeof(float)) {
        R dl[V];
        ldv<R, V>(dl, sa.dz_lo + o);
        F2 qs[V];
#pragma unroll
        for (int x = 0; x < V; ++x) {
          qs[x] = F2{q[0][x], 0.f};
#pragma unroll
          for (int n = 1; n < 5; ++n)
            if (n < nqx) qs[x] = df_add_f(qs[x], q[n][x]);
        }
        for (int n = 5; n < nqx; ++n) {
          ldv<R, V>(q[0], qx + o + (size_t)n * F);
#pragma unroll
          for (int x = 0; x < V; ++x) qs[x] = df_add_f(qs[x], q[0][x]);
        }
#pragma unroll
        for (int x = 0; x < V; ++x)
          if (e + x >= 1 && e + x <= jx - 3) {
            const F2 m = df_mul_f(F2{dz[x], dl[x]}, rh[x]);
            dry2 = df_add(dry2, m);
            qm2 = df_add(qm2, df_mul(m, qs[x]));
          }
      } else {
#pragma unroll
        for (int n = 1; n < 5; ++n)
          if (n < nqx)
#pragma unroll
            for (int x = 0; x < V; ++x) q[0][x] += q[n][x];
        for (int n = 5; n < nqx; ++n) {
          ldv<R, V>(q[1], qx + o + (size_t)n * F);
#pragma unroll
          for (int x = 0; x < V; ++x) q[0][x] += q[1][x];
        }
#pragma unroll
        for (int x = 0; x < V; ++x)
          if (e + x >= 1 && e + x <= jx - 3) {
            const double m = __dmul_rn(dz[x], rh[x]);
            a.dry += m;
            a.qm = __fma_rn(q[0][x], m, a.qm);
          }
      }
    }
    const double dxsq = c.dx * c.dx;
    if constexpr (sizeof(R) == sizeof(float)) {
      a.dry = ((double)dry2.hi + (double)dry2.lo) * dxsq;
      a.qm = ((double)qm2.hi + (double)qm2.lo) * dxsq;
    } else {
      a.dry *= dxsq;
      a.qm *= dxsq;
    }
    // Lateral fluxes, FP64 products of the state's values in both precisions
    // (a few thousand terms: the budget stays FP64-accurate for a mixed
    // member).  wind: into the domain
    auto face = [&](size_t o, double wind) {
      const double f = wind * (sa.dz[o] * (double)st.rho[o]);
      double q = (double)st.qx[o];
      for (int n = 1; n < nqx; ++n) q += (double)st.qx[o + (size_t)n * F];
      a.dadv += f;
      a.qadv = __fma_rn(q, f, a.qadv);
      flux = true;
    };
    // west and east columns over i in ice = 1 .. iy-1 (:85-100)
    for (int e = gt; e < 2 * (iy - 1) * kz; e += gs) {
      const bool east = (e & 1) != 0;
      const int r = e >> 1, k = r / (iy - 1), i = r - k * (iy - 1) + 1;
      const size_t ko = (size_t)k * g.PS;
      const double u = (double)st.u[g.at2(east ? jx : 1, i) + ko];
      face(g.at2(east ? jx - 1 : 1, i) + ko, east ? -u : u);
    }
    // south (v at ide1) and north (v at ide2) rows, j in jci (:101-116)
    for (int e = gt; e < 2 * kz * (jx - 3); e += gs) {
      const int rest = e / (jx - 3), j = e - rest * (jx - 3) + 2;
      const bool north = (rest & 1) != 0;
      const size_t ko = (size_t)(rest >> 1) * g.PS;
      const double v = (double)st.v[g.at2(j, north ? iy : 1) + ko];
      face(g.at2(j, north ? iy - 1 : 1) + ko, north ? -v : v);
    }
    flux = __any_sync(0xffffffffu, flux);
    if (flux) {
      a.dadv *= c.dt * c.dx;
      a.qadv *= c.dt * c.dx;
    }
  }
  // ps and its extrema over the interior
  for (int e = gt; e < (iy - 3) * (jx - 3); e += gs) {
    const int i = e / (jx - 3) + 2, j = e - (i - 2) * (jx - 3) + 2;
    const size_t ij = g.at2(j, i);
    double x;
    if (form_ps) {
      const size_t o1 = ij + (size_t)(kz - 2) * g.PS, o2 = ij + (size_t)(kz - 1) * g.PS;
      x = surface_pressure((double)D.wz[0][o1], (double)D.wz[0][o2], sa.zeta[o1], sa.zeta[o2], (double)st.p[o2]);
      st.ps[ij] = x;
    } else {
      x = st.ps[ij];
    }
    const long long b = __double_as_longlong(x);
    if ((b & 0x7ff0000000000000LL) == 0x7ff0000000000000LL) a.bad = 1;
    else { a.pmax = max(a.pmax, order_key(b)); a.pmin = min(a.pmin, order_key(b)); }
  }
  a = red_block(a, flux, sh);
  if (threadIdx.x == 0) {
    double *p = D.partials + (size_t)blockIdx.x * kNPart;
    p[0] = a.dry; p[1] = a.dadv; p[2] = a.qm; p[3] = a.qadv; 
    p[4] = __longlong_as_double(a.pmax); p[5] = __longlong_as_double(a.pmin); p[6] = a.bad;
    // the member's last block to finish adds the partials: its partials are
    // visible before its ticket, and every other block's before theirs
    __threadfence();
    last = atomicAdd(&D.clk->red_done, 1u) == (unsigned)nb - 1u;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // store the diagnostics, then, where nothing runs beside this, advance the
  // boundary clock and the buffer roles to the next step's, and re-arm the
  // block count
  RedSum t = red_zero();
  for (int b = (int)threadIdx.x; b < nb; b += kRedThreads) {
    const double *p = D.partials + (size_t)b * kNPart;
    t.dry += __ldcg(p); t.dadv += __ldcg(p + 1); t.qm += __ldcg(p + 2); t.qadv += __ldcg(p + 3);
    t.pmax = max(t.pmax, __double_as_longlong(__ldcg(p + 4)));
    t.pmin = min(t.pmin, __double_as_longlong(__ldcg(p + 5)));
    t.bad |= __ldcg(p + 6) != 0.0;
  }
  t = red_block(t, true, sh);
  if (threadIdx.x != 0) return;
  DiagDev *diag = D.diag;
  Clock *clk = D.clk;
  diag->drymass = t.dry; diag->dryadv = t.dadv; diag->qmass = t.qm; diag->qadv = t.qadv;
  diag->ps_max = t.bad ? NAN : __longlong_as_double(order_key(t.pmax));
  diag->ps_min = t.bad ? NAN : __longlong_as_double(order_key(t.pmin));
  diag->nonfinite = t.bad;
  if (t.bad && !clk->nonfinite) { clk->nonfinite = 1; clk->bad_step = clk->step; }
  if (advance) advance_clock(c, clk, uvoff, advoff);
  clk->red_done = 0u;
}

// blockIdx.y: the list's item.  All of an upload's arrays in one launch, after
// their copies: with a kernel after each copy the two engines waited for one
// another (state of 47x33x23: 131 us, 66 so).
__global__ void k_unpack(UnpackList l, Geom g) {
  const UnpackList::Item &t = l.it[blockIdx.y];
  const size_t n = (size_t)t.nj * t.ni * t.nk;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const int j = (int)(e % t.nj);
    const size_t r = e / t.nj;
    const int i = (int)(r % t.ni), k = (int)(r / t.ni);
    const size_t o = (size_t)j + (size_t)i * g.P + (size_t)k * g.PS;
    const double x = t.src[e];
    if (t.f64) {
      static_cast<double *>(t.dst)[o] = x;
    } else {
      // hi = fl(x), lo = fl(x - hi): x to ~48 bits as two floats
      const float hi = (float)x;
      static_cast<float *>(t.dst)[o] = hi;
      if (t.nplane) static_cast<float *>(t.dst)[o + t.nplane] = (float)(x - (double)hi);
    }
  }
}

// What a member keeps derived from the bound 3-D fields, formed where the data
// is: each source crosses the host link once and the host forms no 3-D array
// (binding members of 96x96x30 and 157x157x30: mixed 6.0 ms with these products
// formed on the host, 1.9 so; FP64 16.9 and 2.3).  Every product and quotient
// is rounded by itself.
// Points of the cross grid: the vertical WAF's ratios; mixed members' FP32
// copies, the hydrostatic factor cp*fmzf*dtrdz and dz as a double-float; FP64
// members' factors of the divergence and of the solve.
template <class R>
__global__ void k_bind_cross(Stat<R> sa, Geom g, const double *__restrict__ fmz,
                             const double *__restrict__ fmzf, size_t fp, size_t fps, BindPar b) {
  constexpr bool f64 = sizeof(R) == sizeof(double);
  const size_t nj = (size_t)g.jx - 1, ni = (size_t)g.iy - 1, n = nj * ni * (size_t)(g.kz + 1);
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const size_t j = e % nj, r = e / nj, i = r % ni;
    const int k = (int)(r / ni);
    const size_t o2 = j + i * g.P, o = o2 + (size_t)k * g.PS, f = j + i * fp + (size_t)k * fps;
    const double zf = fmzf[f];
    if constexpr (!f64) {
      const_cast<R *>(sa.fmzf)[o] = (R)zf;
      const double c = __dmul_rn(__dmul_rn(kCpd, zf), b.dtrdz);
      float *cf = reinterpret_cast<float *>(const_cast<double *>(sa.cfz));
      cf[o] = (float)c;
      cf[o + g.PS * (size_t)(g.kz + 1)] = (float)(c - (double)(float)c);
    }
    if (k >= g.kz) continue;
    const double fz = fmz[f];
    const double a = __dmul_rn(b.dtrdz_adv, fz);
    const_cast<R *>(sa.zrfmu)[o] = (R)__ddiv_rn(a, zf);
    const_cast<R *>(sa.zrfmd)[o] = (R)__ddiv_rn(a, fmzf[f + fps]);
    if constexpr (f64) {
      const int ib = sa.ibnd_cr[o2];
      const double bw = ib > 0 ? 1.0 - sa.hefc[(size_t)(ib - 1) + (size_t)k * b.nspgx] : 1.0;
      const_cast<double *>(sa.dv_cf)[o] = __dmul_rn(fz, b.rot ? sa.msfx[o2] : sa.mx2[o2]);
      const_cast<double *>(sa.sv_a)[o] = __dmul_rn(__dmul_rn(bw, b.dtrdz), fz);
      const_cast<double *>(sa.sv_b)[o] = __dmul_rn(b.zcs, fz);
      const_cast<double *>(sa.sv_c)[o] = __dmul_rn(b.dtrdz, fz);
    } else {
      const_cast<R *>(sa.fmz)[o] = (R)fz;
      const double dz = sa.dz[o];
      const_cast<R *>(sa.dz_r)[o] = (R)dz;
      const_cast<R *>(sa.dz_lo)[o] = (R)(dz - (double)(R)dz);
    }
  }
}

// Wind points of an FP64 member: the acoustic substep's constant factors.
__global__ void k_bind_wind(Stat<double> sa, Geom g, BindPar b) {
  const size_t nj = (size_t)g.jx, ni = (size_t)g.iy, n = nj * ni * (size_t)g.kz;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const size_t j = e % nj, r = e / nj, i = r % ni;
    const int k = (int)(r / ni);
    const size_t o2 = j + i * g.P, o = o2 + (size_t)k * g.PS;
    const double gk = sa.gzitakh[k], dk = __dmul_rn(b.dxrdt, sa.xkdamp[k]);
    if (i < ni - 1) {
      const double c = __dmul_rn(b.dtrdx, sa.rfmzu[o]);
      const_cast<double *>(sa.dv_cu)[o] = b.rot ? c : __dmul_rn(c, sa.rmu[o2]);
      const_cast<double *>(sa.mo_gu)[o] = __dmul_rn(__dmul_rn(b.zfz, sa.hx[o2]), gk);
      const_cast<double *>(sa.mo_du)[o] = __dmul_rn(dk, sa.msfu[o2]);
    }
    if (j < nj - 1) {
      const_cast<double *>(sa.dv_cv)[o] = __dmul_rn(__dmul_rn(b.dtrdx, sa.rfmzv[o]), sa.rmv[o2]);
      const_cast<double *>(sa.mo_gv)[o] = __dmul_rn(__dmul_rn(b.zfz, sa.hy[o2]), gk);
      const_cast<double *>(sa.mo_dv)[o] = b.rot ? dk : __dmul_rn(dk, sa.msfv[o2]);
    }
  }
}

template <class R>
__global__ void k_pack3(const R *__restrict__ src, double *__restrict__ dst, Geom g, int nj, int ni, int nk) {
  const size_t n = (size_t)nj * ni * nk;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const int j = (int)(e % nj);
    const size_t r = e / nj;
    const int i = (int)(r % ni);
    const int k = (int)(r / ni);
    dst[e] = (double)src[(size_t)j + (size_t)i * g.P + (size_t)k * g.PS];
  }
}

__global__ void k_pack3_df(const float *__restrict__ src, double *__restrict__ dst, Geom g, int nj,
                           int ni, int nk, size_t nplane) {
  const size_t n = (size_t)nj * ni * nk;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const int j = (int)(e % nj);
    const size_t r = e / nj;
    const int i = (int)(r % ni);
    const int k = (int)(r / ni);
    const size_t o = (size_t)j + (size_t)i * g.P + (size_t)k * g.PS;
    dst[e] = (double)src[o] + (double)src[o + nplane];
  }
}

inline dim3 grid2(int nj, int ni, dim3 b, int nmem) {
  return dim3((unsigned)((nj + b.x - 1) / b.x), (unsigned)((ni + b.y - 1) / b.y), (unsigned)nmem);
}

// grid of a point kernel over nj x ni points per level
inline dim3 pt_grid(const LaunchGeom &L, int nj, int ni, int &tiles_j) {
  tiles_j = (nj + L.col_x - 1) / L.col_x;
  if (L.wl_pt) return dim3((unsigned)L.n_pt, 1, 1);  // one block per work item
  const int ti = (ni + L.col_y - 1) / L.col_y;
  return dim3((unsigned)(tiles_j * ti), (unsigned)((L.kz + L.lv - 1) / L.lv), (unsigned)L.nmem);
}

}  // namespace

// Eight row pieces a warp, at most 2 blocks per SM - a block more costs its
// threads' sums, some 50 FP64 instructions a warp - but down to two pieces a
// warp for the first 64 blocks, whose loads a small domain waits on.  (Of the
// member's extents alone: its sums are the same in any batch.)
int reduce_blocks(const Geom &g) {
  const int items = (g.iy - 3) * g.kz * ((g.jx - 2 + 127) / 128);
  const int eight = (items + 8 * kRedWarps - 1) / (8 * kRedWarps), two = (items + 2 * kRedWarps - 1) / (2 * kRedWarps);
  return std::max(1, std::min(std::max(eight, std::min(two, 64)), 152 * 2));
}

// status_update of the turbulent kinetic energy (Main/mod_moloch.F90:
// 1419-1424): on jci x ici at the kz+1 interfaces, tke + dtsec * tketen (the
// physics' tendency; none in a whole step), then the floor tkemin.
template <class R, int LV>
__global__ void k_end_tke(const Dom<R> *__restrict__ doms, int whole, int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active || !D.c.tke) return;
  const Geom g = D.g;
  const Pt q = point_at<LV>(wi, 1, 1);
  if (q.j < 2 || q.j > g.jx - 2 || q.i < 2 || q.i > g.iy - 2 || q.k > g.kz) return;
  const R *ten = whole ? nullptr : D.tend;
  // tketen follows the kz-plane tendencies (t, u, v, the species, tracers)
  const R *tt = ten ? ten + (size_t)(3 + g.nqx + g.ntr) * g.field3() : nullptr;
  const R dts = pick<R>(D.c.dtsec, D.c.dtsecf);
  const int klast = q.k + LV - 1 >= g.kz ? g.kz + 1 : q.k + LV - 1;
  for (int k = q.k; k <= klast; ++k) {
    const size_t o = g.at(q.j, q.i, k);
    R v = D.tke[o];
    if (tt) v = v + dts * tt[o];
    if (v < R(kTkeMin)) v = R(kTkeMin);
    D.tke[o] = v;
  }
}

template <class R>
void Launch<R>::bdy_ring(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  const unsigned nb = (unsigned)((2 * (L.iy - 2) + 2 * L.jx + kRingThreads - 1) / kRingThreads);
  step_launch(L, k_bdy_ring<R>, dim3(nb, (unsigned)L.kz, (unsigned)L.nmem), kRingThreads, 0, s, d, uvoff, advoff);
}

template <class R>
void Launch<R>::end_relax(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  const dim3 b((unsigned)L.col_x, (unsigned)L.col_y);
  int tj;
  const dim3 grd = pt_grid(L, L.jx - 1, L.iy - 1, tj);
  if (L.lv == 1) step_launch(L, k_end_relax<R, 1>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_pt);
  else step_launch(L, k_end_relax<R, 4>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_pt);
}

template <class R>
void Launch<R>::bdy_spectral(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff,
                             cudaStream_t s) {
  const unsigned fk = (unsigned)(L.kz * 3);
  step_launch(L, k_spec_rows<R>, dim3((unsigned)((L.iy + 7) / 8), fk, (unsigned)L.nmem), 256, 0, s, d, uvoff, advoff);
  step_launch(L, k_spec_modes<R>, dim3(1, fk, (unsigned)L.nmem), 256, 0, s, d);
  const dim3 b((unsigned)L.col_x, (unsigned)L.col_y);
  int tj;
  const dim3 grd = pt_grid(L, L.jx - 2, L.iy - 2, tj);
  if (L.lv == 1) step_launch(L, k_spec_apply<R, 1>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_pt);
  else step_launch(L, k_spec_apply<R, 4>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_pt);
}

template <class R>
void Launch<R>::end_point(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  constexpr int W = 32 * (16 / (int)sizeof(R));
  const int tj = (L.jx - 1 + W - 1) / W, ti = (L.iy - 1 + 3) / 4;
  const dim3 grd = L.wl_vec ? dim3((unsigned)L.n_vec, 1, 1)
                            : dim3((unsigned)(tj * ti), (unsigned)((L.kz + L.lv - 1) / L.lv), (unsigned)L.nmem);
  if (L.lv == 1) step_launch(L, k_end_point<R, 1, false>, grd, 128, 0, s, d, uvoff, advoff, tj, L.wl_vec);
  else step_launch(L, k_end_point<R, 4, false>, grd, 128, 0, s, d, uvoff, advoff, tj, L.wl_vec);
}

template <class R>
void Launch<R>::end_frame(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  const dim3 grd((unsigned)((L.frame_points + 127) / 128), (unsigned)L.kz, (unsigned)L.nmem);
  step_launch(L, k_end_point<R, 1, true>, grd, 128, 0, s, d, uvoff, advoff, 1, nullptr);
}

template <class R>
void Launch<R>::end_uvx(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  const dim3 b((unsigned)L.col_x, (unsigned)L.col_y);
  int tj;
  const dim3 grd = pt_grid(L, L.jx - 1, L.iy - 1, tj);
  if (L.lv == 1) step_launch(L, k_end_uvx<R, 1>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_pt);
  else step_launch(L, k_end_uvx<R, 4>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_pt);
}

template <class R>
void Launch<R>::end_winds(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  const int tj = wind_tiles_j(L.jx), ti = wind_tiles_i(L.iy, L.wind_rows);
  const dim3 grd = L.wl_wind ? dim3((unsigned)L.n_wind, 1, 1)
                             : dim3((unsigned)(tj * ti), (unsigned)L.kz, (unsigned)L.nmem);
  if constexpr (sizeof(R) == sizeof(float))
    step_launch(L, k_end_winds<R>, grd, 32 * kWindWarps, 0, s, d, uvoff, advoff, L.wind_rows, tj, L.wl_wind);
}

template <class R, int PH>
void launch_cross(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  const dim3 b((unsigned)L.col_x, (unsigned)L.col_y);
  int tj;
  const dim3 grd = pt_grid(L, L.jx - 1, L.iy - 1, tj);
  if (PH != kEndPost) step_launch(L, k_end_ps<R>, grid2(L.jx - 3, L.iy - 3, b, L.nmem), b, 0, s, d, uvoff, advoff);
  if (L.lv == 1) step_launch(L, k_end_cross<R, PH, 1>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_pt);
  else step_launch(L, k_end_cross<R, PH, 4>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_pt);
}

template <class R>
void Launch<R>::end_cross(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  if constexpr (sizeof(R) == sizeof(float)) {
    const dim3 b((unsigned)L.col_x, (unsigned)L.col_y), b4(32, 4);
    const int tj = (L.jx - 1 + 127) / 128, ti = (L.iy - 1 + 3) / 4;
    const dim3 grd = L.wl_v4 ? dim3((unsigned)L.n_v4, 1, 1)
                             : dim3((unsigned)(tj * ti), (unsigned)((L.kz + L.lv - 1) / L.lv), (unsigned)L.nmem);
    step_launch(L, k_end_ps<R>, grid2(L.jx - 3, L.iy - 3, b, L.nmem), b, 0, s, d, uvoff, advoff);
    if (L.lv == 1) step_launch(L, k_end_cross_v4<R, 1>, grd, b4, 0, s, d, uvoff, advoff, tj, L.wl_v4);
    else step_launch(L, k_end_cross_v4<R, 4>, grd, b4, 0, s, d, uvoff, advoff, tj, L.wl_v4);
  } else {
    launch_cross<R, kEndAll>(L, d, uvoff, advoff, s);
  }
}

template <class R>
void Launch<R>::end_cross_split(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, bool post,
                                cudaStream_t s) {
  if (post) launch_cross<R, kEndPost>(L, d, uvoff, advoff, s);
  else launch_cross<R, kEndPre>(L, d, uvoff, advoff, s);
}

template <class R>
void Launch<R>::end_uvstag(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  const dim3 b((unsigned)L.col_x, (unsigned)L.col_y);
  int tj;
  const dim3 grd = pt_grid(L, L.jx, L.iy, tj);
  if (L.lv == 1) step_launch(L, k_end_uvstag<R, 1>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_pt);
  else step_launch(L, k_end_uvstag<R, 4>, grd, b, 0, s, d, uvoff, advoff, tj, L.wl_pt);
}

template <class R>
void Launch<R>::end_tke(const LaunchGeom &L, const Dom<R> *d, bool whole_step, cudaStream_t s) {
  const dim3 b((unsigned)L.col_x, (unsigned)L.col_y);
  int tj;
  const dim3 grd = pt_grid(L, L.jx, L.iy, tj);
  if (L.lv == 1) step_launch(L, k_end_tke<R, 1>, grd, b, 0, s, d, whole_step ? 1 : 0, tj, L.wl_pt);
  else step_launch(L, k_end_tke<R, 4>, grd, b, 0, s, d, whole_step ? 1 : 0, tj, L.wl_pt);
}

template <class R>
void Launch<R>::end_reduce(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, bool form_ps, bool advance,
                           cudaStream_t s) {
  step_launch(L, k_reduce_partial<R>, dim3((unsigned)L.red_blocks, (unsigned)L.nmem), kRedThreads, 0, s, d, uvoff,
              advoff, form_ps ? 1 : 0, advance ? 1 : 0);
}

template <class R>
void Launch<R>::end_advance(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s) {
  step_launch(L, k_end_advance<R>, (unsigned)((L.nmem + 63) / 64), 64, 0, s, d, L.nmem, uvoff, advoff);
}

template <class R>
void Launch<R>::bind_derived(const Stat<R> &sa, const Geom &g, const double *fmz, const double *fmzf,
                             size_t fp, size_t fps, const BindPar &b, cudaStream_t s) {
  k_bind_cross<R><<<152 * 8, 256, 0, s>>>(sa, g, fmz, fmzf, fp, fps, b);
  if constexpr (sizeof(R) == sizeof(double)) k_bind_wind<<<152 * 8, 256, 0, s>>>(sa, g, b);
}

template <class R>
void Launch<R>::unpack(const UnpackList &l, const Geom &g, cudaStream_t s) {
  k_unpack<<<dim3((unsigned)(152 * 8 / l.n + 1), (unsigned)l.n), 256, 0, s>>>(l, g);
}

template <class R>
void Launch<R>::pack3(const R *src, double *dst, const Geom &g, int nj, int ni, int nk, cudaStream_t s) {
  k_pack3<R><<<152 * 8, 256, 0, s>>>(src, dst, g, nj, ni, nk);
}

template <class R>
void Launch<R>::pack3_df(const double *src, double *dst, const Geom &g, int nj, int ni, int nk,
                         size_t nplane, cudaStream_t s) {
  k_pack3_df<<<152 * 8, 256, 0, s>>>(reinterpret_cast<const float *>(src), dst, g, nj, ni, nk, nplane);
}

template struct Launch<double>;
template struct Launch<float>;

}  // namespace mlc
