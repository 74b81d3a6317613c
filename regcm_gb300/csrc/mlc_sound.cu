// mlc_sound.cu -- the acoustic substeps of the MOLOCH step
// (Main/mod_moloch.F90:531-765, subroutines sound, divergence_damping,
// divergence_diffusion).
//
// One substep is three kernels:
//   sound_div       per column of cross points: raw horizontal divergence
//                   zdiv2 (Eq. 16) and the generalized vertical velocity s
//                   (Eq. 10), s(kz+1) and the surface w.
//   sound_solve     per interior column: the 5-point divergence filter, the
//                   vertical divergence term, the implicit w-Exner tridiagonal
//                   system (Eq. 19, Thomas algorithm), the Exner update and,
//                   after the last substep, the completed s.  A column is one
//                   thread's, streamed through shared memory, or several warps'
//                   and kept on chip (solve_form).
//   sound_momentum  u and v (Eq. 17/18): divergence damping, Coriolis with
//                   the substep's initial winds, pressure gradient with the new
//                   Exner function, terrain term, relaxation-zone weight.  It
//                   writes the other half of a ping-pong pair, which is how the
//                   reference's ud/vd copies are kept without a copy.
// theta_v does not change during the substeps, so what it enters is formed
// once a round by sound_prep: the solve's hydrostatic factor Z =
// cp*theta_v(half)*fmzf*dtrdz with its decrement per unit w, and the
// momentum's pressure-gradient coefficients.  Departures from the reference's
// operand order: those factors, FMA contraction, and the relaxation weight
// bdywt recomputed from ibnd and hefc instead of read from an array (the same
// value, Main/mod_bdycod.F90:4033-4047).
#include "mlc_kernels.cuh"
#include "mlc_tma.cuh"

namespace mlc {

namespace {

// The scratch planes of the acoustic loop (the WAF's wz planes, free then).
// FP64: the filtered divergence and the multipliers between the solve's two
// passes, then G, Cu, Cv.  Mixed: those two are double-float planes (wz_d),
// and there is no Cu, Cv.
template <class R>
struct SoundScratch {
  R *zf, *mul, *g, *cu, *cv;
  R *w_lo, *mul_lo;  // mixed: low parts of the eliminated w and the multipliers
};
template <class R>
__device__ __forceinline__ SoundScratch<R> sound_scratch(const Dom<R> &D) {
  if constexpr (sizeof(R) == sizeof(double)) {
    return {D.wz[0], D.wz[1], D.wz[2], D.wz[3], D.wz[4], nullptr, nullptr};
  } else {
    float *zf = reinterpret_cast<float *>(D.wz_d[0]), *mul = reinterpret_cast<float *>(D.wz_d[1]);
    return {zf, mul, D.wz[2], nullptr, nullptr, zf + D.g.field3(), mul + D.g.field3()};
  }
}

__device__ __forceinline__ double relax_weight(const int32_t *ibnd, const double *hefc, int nsp,
                                               size_t ij, int k) {
  int ib = ibnd[ij];
  return ib > 0 ? 1.0 - hefc[(size_t)(ib - 1) + (size_t)(k - 1) * nsp] : 1.0;
}

// What the substeps of one advection round read of theta_v (constant over
// them), at cross point (j, i), level k:
//   Z(k)  = theta_v(half) * cp*fmzf*dtrdz, k = 2..kz (:564-566 with the
//           factor of :641), which the solves lower by w*G every substep
//   G(k)  = (fmzf*dtrdz)*(theta_v(k-1) - theta_v(k)) * cp*fmzf*dtrdz
//   Cu, Cv = zcx*cp/2*(theta_v sum) of the momentum's pressure gradients
//           (an FP64 member's)
// in tetavf and the scratch planes the solves leave free.  Per substep this
// takes six FP64 instructions a point out of the momentum and nine out of the
// solve for thirteen here once a round; in the mixed solve a double-float
// product and 12 bytes a point.  A mixed member's momentum, bound by memory,
// reads theta_v itself: two coefficient planes would be as many bytes and cost
// their writing here (measured 353 + 92 against 366 + 73 us a step of four
// substeps at 512x512x41).
template <class R, int LV>
__global__ void k_sound_prep(const Dom<R> *__restrict__ doms, int advoff, int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const Pt q = point_at<LV>(wi, 1, 1);
  if (q.j > g.jx - 1 || q.i > g.iy - 1 || q.k > g.kz) return;
  const int adv = (D.clk->adv_role + advoff) & 1;
  const Scal &c = D.c;
  const Stat<R> &sa = D.sa;
  const double *__restrict__ tetav = D.tetav[adv];
  const SoundScratch<R> ss = sound_scratch(D);
  const size_t ij = g.at2(q.j, q.i), S = (size_t)g.P;
  double cx = 0.0, cy = 0.0;
  if constexpr (sizeof(R) == sizeof(double)) {
    cx = c.dtrdxs * sa.msfu[ij] * (0.5 * kCpd);
    cy = (c.lrotllr ? c.dtrdxs : c.dtrdxs * sa.msfv[ij]) * (0.5 * kCpd);
  }
#pragma unroll
  for (int k = q.k; k < q.k + LV && k <= g.kz; ++k) {
    const size_t o = g.at(q.j, q.i, k), om = o - g.PS;
    if constexpr (sizeof(R) == sizeof(float)) {
      const DF th(tetav, g.field3()), zz(D.tetavf, g.PS * (size_t)(g.kz + 1));
      if (k < 2) continue;
      const F2 tm = th.ld(om), t0 = th.ld(o);
      const F2 sm = df_add(tm, t0);
      const F2 cf = DF(sa.cfz, g.PS * (size_t)(g.kz + 1)).ld(o);
      zz.st(o, df_mul(F2{0.5f * sm.hi, 0.5f * sm.lo}, cf));
      ss.g[o] = sa.fmzf[o] * (c.dtsoundf * c.rdzitaf) * df_diff(tm, t0) * df_f(cf);
    } else {
      const double t0 = tetav[o];
      if (q.j >= 2) ss.cu[o] = cx * (tetav[o - 1] + t0);
      if (q.i >= 2) ss.cv[o] = cy * (tetav[o - S] + t0);
      if (k < 2) continue;
      const double tm = tetav[om], fd = sa.fmzf[o] * (c.dtsound * c.rdzita), cf = kCpd * fd;
      D.tetavf[o] = (0.5 * (tm + t0)) * cf;
      ss.g[o] = (fd * (tm - t0)) * cf;
    }
  }
}

// zdiv2 (Main/mod_moloch.F90:602-618) from the face fluxes u*cu and v*cv, and
// the terrain-following wind of s (:582-597) from the winds summed over two
// levels; every rounding explicit (the chunk sizes of the point kernels give
// the same bits).
template <class R>
__device__ __forceinline__ R divergence(R cf, R u0, R cu0, R u1, R cu1, R v0, R cv0, R v1, R cv1) {
  return mul_r(cf, fma_r(-v0, cv0, fma_r(v1, cv1, fma_r(u1, cu1, -mul_r(u0, cu0)))));
}
template <class R>
__device__ __forceinline__ R slope_wind(R u0, R hx0, R u1, R hx1, R v0, R hy0, R v1, R hy1) {
  return fma_r(v1, hy1, fma_r(v0, hy0, fma_r(u1, hx1, mul_r(u0, hx0))));
}

// Main/mod_moloch.F90:582-618, FP64.  Bound by the FP64 pipe: 14 instructions
// a point (17 with the reference's association).
template <class R, int LV>
__global__ void k_sound_div(const Dom<R> *__restrict__ doms, int uvoff, int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  static_assert(sizeof(R) == sizeof(double), "FP64 member");
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const Pt q = point_at<LV>(wi, 1, 1);
  const int j = q.j, i = q.i, kz = g.kz;
  if (j > g.jx - 1 || i > g.iy - 1 || q.k > kz) return;
  const Stat<R> &sa = D.sa;
  const int uv = (D.clk->uv_role + uvoff) & 1;
  const R *__restrict__ u = D.u[uv];
  const R *__restrict__ v = D.v[uv];
  R *__restrict__ zdiv2 = D.zdiv2;
  R *__restrict__ s = D.s;
  R *__restrict__ w = D.w;
  const size_t ij = g.at2(j, i), ijE = g.at2(j + 1, i), ijN = g.at2(j, i + 1);
  const bool interior = (j >= 2 && j <= g.jx - 2 && i >= 2 && i <= g.iy - 2);
  R hx0 = 0, hx1 = 0, hy0 = 0, hy1 = 0;
  if (interior) {
    hx0 = sa.hx[ij]; hx1 = sa.hx[ijE]; hy0 = sa.hy[ij]; hy1 = sa.hy[ijN];
  }
#pragma unroll
  for (int k = q.k; k < q.k + LV && k <= kz; ++k) {
    const size_t o = (size_t)(k - 1) * g.PS;
    const R u0 = u[ij + o], u1 = u[ijE + o], v0 = v[ij + o], v1 = v[ijN + o];
    // the constant factors formed at bind time
    zdiv2[ij + o] = divergence<R>(sa.dv_cf[ij + o], u0, sa.dv_cu[ij + o], u1, sa.dv_cu[ijE + o], v0,
                                  sa.dv_cv[ij + o], v1, sa.dv_cv[ijN + o]);
    if (!interior) continue;
    if (k >= 2) {
      const size_t om = o - g.PS;  // level k-1
      s[ij + o] = mul_r(slope_wind<R>(u0 + u[ij + om], hx0, u1 + u[ijE + om], hx1, v0 + v[ij + om], hy0,
                                      v1 + v[ijN + om], hy1),
                        sa.gzitak[k - 1]);
    }
    if (k == kz) {
      const R skp1 = -0.5 * slope_wind<R>(u0, hx0, u1, hx1, v0, hy0, v1, hy1);
      s[ij + (size_t)kz * g.PS] = skp1;
      w[ij + (size_t)kz * g.PS] = -skp1;
    }
  }
}

// Two forms of each solve, picked by the number of column segments
// (solve_form).  Their level arithmetic is the functions below, every rounding
// explicit, so the forms agree bit for bit: a member's result does not depend
// on what else a launch holds.
//
// FP64 (Main/mod_moloch.F90:627-671).  The FP64 instructions bound the large
// grids, so the arithmetic is arranged for few of them: with Z =
// cp*theta_v(half)*fmzf*dtrdz (sound_prep) lowered by w*G,
//   w_expl = w - Z*(dpai - R/cv*d(pai*zf)) - g*dts,   d = (m) - (k) = above - below
//   zu, zd = Z*(b*pai) + ffilt,                       b = dtrdz*R/cv*fmz
// with pai*zf and b*pai of a level formed once and carried to the next: 31 a
// column and level, against 47 for the reference's own association.
struct LevelD {
  double s, pai, zf, pz, bp;  // pz: pai*zf, bp: b*pai
};
// z: the raw divergence here, w/e/s/n its neighbours (:531-543); fza:
// (bw*dtrdz)*fmz; ds: s here minus s below (:627-630)
__device__ __forceinline__ void level_d(LevelD &v, bool filt, double xk, double z, double zw, double ze, double zs,
                                        double zn, double fza, double ds, double fzb) {
  if (filt) z = __fma_rn(xk, __fma_rn(-4.0, z, zw + ze + zs + zn), z);
  v.zf = __fma_rn(fza, ds, z);
  v.pz = __dmul_rn(v.pai, v.zf);
  v.bp = __dmul_rn(fzb, v.pai);
}
struct CoefD {
  double zw, zd, zu, den;  // w_expl; den: 1 + zd + zu
};
__device__ __forceinline__ CoefD coef_d(const LevelD &vm, const LevelD &vk, double Z, double wold, double ff,
                                        double gdts) {
  // the hydrostatic balance -Z*dpai - g*dts in one fused multiply-add
  const double e = __fma_rn(-kRdrcv, __dsub_rn(vm.pz, vk.pz), vm.pai - vk.pai);
  CoefD c;
  c.zw = __dadd_rn(wold, __fma_rn(-Z, e, -gdts));
  c.zu = __fma_rn(vm.bp, Z, ff);
  c.zd = __fma_rn(vk.bp, Z, ff);
  c.den = __dadd_rn(__dadd_rn(1.0, c.zd), c.zu);
  return c;
}
// one level of the elimination: the eliminated w and the multiplier
__device__ __forceinline__ void eliminate_d(double &w, double &mul, const CoefD &c) {
  const double r = recip_d(__fma_rn(-c.zd, mul, c.den));
  w = __dmul_rn(r, __fma_rn(c.zd, w, c.zw));
  mul = __dmul_rn(r, c.zu);
}
__device__ __forceinline__ double exner_d(double pai, double zf, double fzc, double w, double wbelow) {
  return __dmul_rn(pai, __fma_rn(-kRdrcv, __fma_rn(fzc, __dsub_rn(w, wbelow), zf), 1.0));
}

// Mixed members, in FP32 only.  Where rounding is amplified the values are
// double-floats: Z, the hydrostatic balance -Z*(pai(k-1) - pai(k)) - g*dts of
// the w equation (two terms of ~g*dts whose difference drives w), the Exner
// update pai - pai*increment and, with DFR, the recurrence.  The divergence
// filter and the elimination coefficients (O(1)-conditioned) run in plain FP32.
struct LevelF {
  float s, zf, fp, pz;  // fp: dtrdz*fmz*pai, pz: pai*zf
  F2 pai;
};
__device__ __forceinline__ void level_f(LevelF &v, bool filt, float xk, float z, float zw, float ze, float zs,
                                        float zn, float bw, float fz, float ds) {
  if (filt) z = fmaf(xk, fmaf(-4.f, z, zw + ze + zs + zn), z);
  v.zf = fmaf(__fmul_rn(bw, fz), ds, z);
  const float p = df_f(v.pai);
  v.fp = __fmul_rn(fz, p);
  v.pz = __fmul_rn(p, v.zf);
}
struct CoefF {
  F2 zw;
  float zd, zu;
};
__device__ __forceinline__ CoefF coef_f(const LevelF &vm, const LevelF &vk, F2 Z, float wold, float ff, F2 ngdts) {
  const F2 dp = two_sum(vm.pai.hi - vk.pai.hi, vm.pai.lo - vk.pai.lo);
  const F2 bal = df_add(ngdts, df_mul(F2{-Z.hi, -Z.lo}, dp));
  const float zr = __fmul_rn(float(kRdrcv), df_f(Z));
  CoefF c;
  c.zw = df_add_f(df_add_f(bal, wold), __fmul_rn(zr, __fsub_rn(vm.pz, vk.pz)));
  c.zu = fmaf(zr, vm.fp, ff);
  c.zd = fmaf(zr, vk.fp, ff);
  return c;
}
// (den >= 1: the pivot of a diagonally dominant system)
template <bool DFR>
__device__ __forceinline__ void eliminate_f(F2 &w, F2 &mul, const CoefF &c) {
  if constexpr (DFR) {
    const F2 den = df_add(two_sum(__fadd_rn(1.f, c.zd), c.zu), df_mul_f(F2{-mul.hi, -mul.lo}, c.zd));
    const F2 r = df_recip(den);
    w = df_mul(r, df_add(c.zw, df_mul_f(w, c.zd)));
    mul = df_mul_f(r, c.zu);
  } else {
    const float r = 1.f / fmaf(-c.zd, mul.hi, __fadd_rn(__fadd_rn(1.f, c.zd), c.zu));
    w.hi = __fmul_rn(r, fmaf(c.zd, w.hi, df_f(c.zw)));
    mul.hi = __fmul_rn(r, c.zu);
  }
}
template <bool DFR>
__device__ __forceinline__ F2 back_f(F2 wel, F2 mul, F2 wabove) {
  if constexpr (DFR) return df_add(wel, df_mul(mul, wabove));
  else return F2{fmaf(mul.hi, wabove.hi, wel.hi), 0.f};
}
// dzf: dtrdz*fmz
__device__ __forceinline__ F2 exner_f(F2 pai, float zf, float dzf, F2 w, F2 wbelow) {
  const float inc = __fmul_rn(float(kRdrcv), fmaf(dzf, df_diff(w, wbelow), zf));
  const F2 d = df_mul_f(pai, inc);
  return df_add(pai, F2{-d.hi, -d.lo});
}

// ---- the solves, a column by several warps ------------------------------------
// A block is 32 columns of a row (lanes are columns).  AW warps form the
// coefficients, kSolveLevels interfaces in turn each, and leave them in shared
// memory; one warp runs the elimination behind them, an mbarrier a round
// telling it that the round's coefficients are there.  The column stays on
// chip: the back substitution overwrites the eliminated values, and all warps
// update Exner (and s after the last substep) level by level.  The elimination
// warp's place rotates with the block, so that the SM's four schedulers get it
// equally often.
//
// Why: on GB300 an FP64 instruction of a warp takes 64 clocks of its scheduler's FP64
// unit, however many lanes are active, and a column's elimination is a serial
// chain; with one warp a segment three of an SM's four units idle unless many
// segments share the SM, and the mixed solve is a chain of double-float
// operations the same way.
constexpr int kSolveCols = 32;
// interfaces a coefficient warp forms a round (a round's first level costs the
// filtered divergence once more; 1 and 4 measured slower)
constexpr int kSolveLevels = 2;
// threads of a block: with six coefficient warps two share each scheduler but
// the elimination's, whose second warp only joins the Exner update
constexpr int solve_threads(int aw) { return 32 * (aw > 3 ? 8 : 4); }

// This thread's part of a block: its role (0 eliminates, 1..AW coefficients,
// AW+1 of the six-warp form only the Exner update)
// and its column; lanes outside the interior work on the nearest interior
// column and store nothing.
struct SolveLane {
  int role, lane, col;  // col: j - 1
  bool act;
};
template <int AW>
__device__ __forceinline__ SolveLane solve_lane(const Geom &g, int x0) {
  SolveLane l;
  l.lane = (int)threadIdx.x & 31;
  const int wp = (int)threadIdx.x >> 5;
  // warps p and p+4 share a scheduler: the eliminating warp's is left to it
  const int q = (wp + (int)(blockIdx.x + blockIdx.y)) & 3;
  l.role = q == 0 ? (wp < 4 ? 0 : AW + 1) : wp < 4 ? q : q + 3;
  const int j = x0 + l.lane + 1;
  l.act = j >= 2 && j <= g.jx - 2;
  l.col = min(max(j, 2), g.jx - 2) - 1;
  return l;
}

// FP64 members (s :728-734).
template <class R, int AW>
__global__ void __launch_bounds__(solve_threads(AW), 512 / solve_threads(AW)) k_solve_cols_d(const Dom<R> *__restrict__ doms, int advoff,
                                                                  int last, const WorkItem *__restrict__ wl) {
  grid_begin();
  static_assert(sizeof(R) == sizeof(double), "FP64 member");
  constexpr int NL = kSolveLevels, NR = AW * NL;  // interfaces a warp, a round
  extern __shared__ __align__(16) double dv_smem[];
  __shared__ __align__(8) uint64_t mbar[kMaxLevels / NR + 1];  // a round's coefficients are there
  const WorkItem wi = wl ? wl[blockIdx.x]
                          : WorkItem{(int16_t)blockIdx.z, (int16_t)blockIdx.x, (int16_t)blockIdx.y, 0};
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const int x0 = (int)wi.a * kSolveCols, i = (int)wi.b + 2;
  if (x0 + 1 > g.jx - 2 || i > g.iy - 2) return;  // uniform over the block
  const SolveLane l = solve_lane<AW>(g, x0);
  const int kz = g.kz, PS = (int)g.PS, P = g.P;
  if ((int)threadIdx.x <= kMaxLevels / NR) {
    mbar_init(&mbar[threadIdx.x], AW);
    fence_mbar_init();
  }
  __syncthreads();
  const Scal &c = D.c;
  const Stat<R> &sa = D.sa;
  const int adv = (D.clk->adv_role + advoff) & 1;
  const size_t r0 = g.at2(1, i) + (size_t)l.col;
  const double *__restrict__ zraw = D.zdiv2 + r0;
  const double *__restrict__ fza = sa.sv_a + r0;
  const double *__restrict__ fzb = sa.sv_b + r0;
  const double *__restrict__ gg = sound_scratch(D).g + r0;
  double *__restrict__ s = D.s + r0;
  double *__restrict__ w = D.w + r0;
  double *__restrict__ pai = D.pai[adv] + r0;
  double *__restrict__ zp = D.tetavf + r0;
  const bool filt = c.divfilter != 0;
  // rows k = 0 .. kz+1 of 32 columns: 1 + zd + zu; zd; zu, then the
  // multiplier; w_expl, then the eliminated w, then w; filtered divergence
  const int rows = (kz + 2) * 32;
  double *sa_ = dv_smem + l.lane, *sd = sa_ + rows, *su = sd + rows, *sw = su + rows, *sf = sw + rows;
  auto level = [&](int m, double s_below, bool keep) {
    const int o = (m - 1) * PS;
    LevelD v;
    v.s = s[o];
    v.pai = pai[o];
    const double z = zraw[o];
    if (filt)
      level_d(v, true, sa.xknu[m - 1], z, zraw[o - 1], zraw[o + 1], zraw[o - P], zraw[o + P], fza[o], v.s - s_below,
              fzb[o]);
    else
      level_d(v, false, 0.0, z, 0.0, 0.0, 0.0, 0.0, fza[o], v.s - s_below, fzb[o]);
    if (keep) sf[m * 32] = v.zf;
    return v;
  };
  const double gdts = kGrav * c.dtsound;
  double wnext = 0.0, wkp1 = 0.0;
  if (l.role == 0) {
    wnext = w[kz * PS];  // w(kz+1) = -s(kz+1)
    sw[(kz + 1) * 32] = wnext;
    sw[32] = w[0];       // w(1) = 0
  }
  const int nr = (kz - 1 + NR - 1) / NR;
  bool ok = true;
  if (l.role >= 1 && l.role <= AW) {
    for (int r = 0; r < nr; ++r) {
      const int kt = kz - r * NR - (l.role - 1) * NL;  // this warp's first interface
      if (kt >= 2) {
        LevelD vk = level(kt, s[kt * PS], kt == kz);
#pragma unroll
        for (int n = 0; n < NL; ++n) {
          const int k = kt - n;
          if (k < 2) break;
          const int o = (k - 1) * PS;
          const double wold = w[o];
          const LevelD vm = level(k - 1, vk.s, true);
          const double Z = __fma_rn(-wold, gg[o], zp[o]);
          if (l.act) zp[o] = Z;
          const CoefD cf = coef_d(vm, vk, Z, wold, sa.ffilt[k - 1], gdts);
          sw[k * 32] = cf.zw;
          sd[k * 32] = cf.zd;
          su[k * 32] = cf.zu;
          sa_[k * 32] = cf.den;
          vk = vm;
        }
      }
      __syncwarp();
      if (l.lane == 0) mbar_arrive(&mbar[r]);
    }
  } else if (l.role == 0) {
    for (int r = 0; r < nr && ok; ++r) {
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(&mbar[r], 0u));
      const int k0 = kz - r * NR, k1 = max(2, k0 - NR + 1);
      for (int k = k0; k >= k1; --k) {
        eliminate_d(wnext, wkp1, CoefD{sw[k * 32], sd[k * 32], su[k * 32], sa_[k * 32]});
        sw[k * 32] = wnext;
        su[k * 32] = wkp1;
      }
    }
    double wp = sw[32];
    for (int k = 2; k <= kz; ++k) {
      wp = __fma_rn(su[k * 32], wp, sw[k * 32]);
      sw[k * 32] = wp;
      if (l.act) w[(k - 1) * PS] = wp;
    }
  }
  if (__syncthreads_or(!ok)) {
    if (threadIdx.x == 0) atomicOr(&D.clk->fault, 1);
    return;
  }
  if (!l.act) return;
  // Exner (:668-671) and s (:728-734), a level a warp
  const double *__restrict__ fzc = sa.sv_c + r0;
  const double *__restrict__ fzf = sa.fmzf_d + r0;
#pragma unroll 3
  for (int m = 1 + l.role; m <= kz; m += solve_threads(AW) / 32) {
    const int o = (m - 1) * PS;
    const double wm = sw[m * 32];
    pai[o] = exner_d(pai[o], sf[m * 32], fzc[o], wm, sw[(m + 1) * 32]);
    if (last) s[o] = m >= 2 ? (wm + s[o]) * fzf[o] : 0.0;
  }
  if (last && l.role == 0) s[kz * PS] = 0.0;
}

// Mixed members.
template <class R, int AW, bool DFR>
__global__ void __launch_bounds__(solve_threads(AW), 1024 / solve_threads(AW)) k_solve_cols_f(const Dom<R> *__restrict__ doms, int advoff,
                                                                  int last, const WorkItem *__restrict__ wl) {
  grid_begin();
  static_assert(sizeof(R) == sizeof(float), "FP32 fields");
  constexpr int NL = kSolveLevels, NR = AW * NL;
  extern __shared__ __align__(16) float sv_smem[];
  __shared__ __align__(8) uint64_t mbar[kMaxLevels / NR + 1];
  const WorkItem wi = wl ? wl[blockIdx.x]
                          : WorkItem{(int16_t)blockIdx.z, (int16_t)blockIdx.x, (int16_t)blockIdx.y, 0};
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const int x0 = (int)wi.a * kSolveCols, i = (int)wi.b + 2;
  if (x0 + 1 > g.jx - 2 || i > g.iy - 2) return;  // uniform over the block
  const SolveLane l = solve_lane<AW>(g, x0);
  const int kz = g.kz, PS = (int)g.PS, P = g.P;
  if ((int)threadIdx.x <= kMaxLevels / NR) {
    mbar_init(&mbar[threadIdx.x], AW);
    fence_mbar_init();
  }
  __syncthreads();
  const Scal &c = D.c;
  const Stat<R> &sa = D.sa;
  const int adv = (D.clk->adv_role + advoff) & 1;
  const unsigned F = (unsigned)g.field3(), F1 = F + (unsigned)PS;
  const size_t r0 = g.at2(1, i) + (size_t)l.col;
  const float *__restrict__ zraw = D.zdiv2 + r0;
  const float *__restrict__ fmz = sa.fmz + r0;
  const float *__restrict__ gg = sound_scratch(D).g + r0;
  float *__restrict__ s = D.s + r0;
  float *__restrict__ w = D.w + r0;
  float *__restrict__ pai = reinterpret_cast<float *>(D.pai[adv]) + r0;
  float *__restrict__ zp = reinterpret_cast<float *>(D.tetavf) + r0;
  const float dtrdz = c.dtsoundf * c.rdzitaf;
  const bool filt = c.divfilter != 0;
  const int32_t ib = sa.ibnd_cr[r0];
  // rows k = 0 .. kz+1 of 32 columns: zd, then the multiplier's low part; zu,
  // then the multiplier; w_expl, then the eliminated w, then w (low part; high
  // part); filtered divergence
  const int rows = (kz + 2) * 32;
  float *sd = sv_smem + l.lane, *su = sd + rows, *swl = su + rows, *sw = swl + rows, *sf = sw + rows;
  auto level = [&](int m, float s_below, bool keep) {
    const int o = (m - 1) * PS;
    LevelF v;
    v.s = s[o];
    v.pai = F2{pai[o], pai[o + F]};
    const float z = zraw[o], fz = __fmul_rn(dtrdz, fmz[o]);
    const float bw = ib > 0 ? 1.f - sa.hefc_r[(size_t)(ib - 1) + (size_t)(m - 1) * c.nspgx] : 1.f;
    if (filt)
      level_f(v, true, sa.xknu_r[m - 1], z, zraw[o - 1], zraw[o + 1], zraw[o - P], zraw[o + P], bw, fz, v.s - s_below);
    else
      level_f(v, false, 0.f, z, 0.f, 0.f, 0.f, 0.f, bw, fz, v.s - s_below);
    if (keep) sf[m * 32] = v.zf;
    return v;
  };
  const F2 ngdts{-c.gdts_hi, -c.gdts_lo};
  F2 wnext{0.f, 0.f}, wkp1{0.f, 0.f};
  if (l.role == 0) {
    wnext.hi = w[kz * PS];
    sw[(kz + 1) * 32] = wnext.hi;
    swl[(kz + 1) * 32] = 0.f;
    sw[32] = w[0];
    swl[32] = 0.f;
  }
  const int nr = (kz - 1 + NR - 1) / NR;
  bool ok = true;
  if (l.role >= 1 && l.role <= AW) {
    for (int r = 0; r < nr; ++r) {
      const int kt = kz - r * NR - (l.role - 1) * NL;
      if (kt >= 2) {
        LevelF vk = level(kt, s[kt * PS], kt == kz);
#pragma unroll
        for (int n = 0; n < NL; ++n) {
          const int k = kt - n;
          if (k < 2) break;
          const int o = (k - 1) * PS;
          const float wold = w[o];
          const LevelF vm = level(k - 1, vk.s, true);
          const F2 Z = df_add_f(F2{zp[o], zp[o + F1]}, -__fmul_rn(wold, gg[o]));
          if (l.act) {
            zp[o] = Z.hi;
            zp[o + F1] = Z.lo;
          }
          const CoefF cf = coef_f(vm, vk, Z, wold, sa.ffilt_r[k - 1], ngdts);
          sd[k * 32] = cf.zd;
          su[k * 32] = cf.zu;
          sw[k * 32] = cf.zw.hi;
          swl[k * 32] = cf.zw.lo;
          vk = vm;
        }
      }
      __syncwarp();
      if (l.lane == 0) mbar_arrive(&mbar[r]);
    }
  } else if (l.role == 0) {
    for (int r = 0; r < nr && ok; ++r) {
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(&mbar[r], 0u));
      const int k0 = kz - r * NR, k1 = max(2, k0 - NR + 1);
      for (int k = k0; k >= k1; --k) {
        eliminate_f<DFR>(wnext, wkp1, CoefF{F2{sw[k * 32], swl[k * 32]}, sd[k * 32], su[k * 32]});
        sw[k * 32] = wnext.hi;
        swl[k * 32] = wnext.lo;
        su[k * 32] = wkp1.hi;
        sd[k * 32] = wkp1.lo;
      }
    }
    F2 wp{sw[32], 0.f};
    for (int k = 2; k <= kz; ++k) {
      wp = back_f<DFR>(F2{sw[k * 32], swl[k * 32]}, F2{su[k * 32], sd[k * 32]}, wp);
      sw[k * 32] = wp.hi;
      swl[k * 32] = wp.lo;
      if (l.act) w[(k - 1) * PS] = df_f(wp);
    }
  }
  if (__syncthreads_or(!ok)) {
    if (threadIdx.x == 0) atomicOr(&D.clk->fault, 1);
    return;
  }
  if (!l.act) return;
#pragma unroll 3
  for (int m = 1 + l.role; m <= kz; m += solve_threads(AW) / 32) {
    const int o = (m - 1) * PS;
    const F2 pp{pai[o], pai[o + F]}, wm{sw[m * 32], swl[m * 32]};
    const F2 pn = exner_f(pp, sf[m * 32], __fmul_rn(dtrdz, fmz[o]), wm, F2{sw[(m + 1) * 32], swl[(m + 1) * 32]});
    pai[o] = pn.hi;
    pai[o + F] = pn.lo;
    if (last) s[o] = m >= 2 ? (df_f(wm) + s[o]) * sa.fmzf[r0 + o] : 0.f;
  }
  if (last && l.role == 0) s[kz * PS] = 0.f;
}

// ---- the solves, streamed: one thread a column --------------------------------
// Where the grid fills the GPU (solve_form).
// A block is a row segment of CW columns (one thread a column).  The downward
// pass forms each level's coefficients and eliminates at once, the upward pass
// substitutes back and updates Exner (and s after the last substep) a level
// behind.  Every level's planes arrive in shared memory as row segments by
// untiled bulk copies kStages levels ahead of the level being solved (the raw
// divergence with a halo); the lanes of warp 0 issue them, one plane a lane,
// each lane keeping its plane's address.  Between the passes the eliminated w
// stays in w, the multipliers and the filtered divergence in scratch planes.
//
// Shared layout of a stage, in elements: three rows of the raw divergence
// (i, i-1, i+1; kHalo columns either side, which keeps 16-byte alignment),
// then kPlanes rows of CW.  The upward pass uses the divergence rows for its
// last two planes.
template <class R, int CW>
struct SolveShape {
  static constexpr bool kF64 = sizeof(R) == sizeof(double);
  static constexpr int kHalo = 16 / (int)sizeof(R) > 2 ? 16 / (int)sizeof(R) : 2;
  static constexpr int kZW = CW + 2 * kHalo;
  static constexpr int kPlanes = kF64 ? 7 : 8;
  static constexpr int kStage = 3 * kZW + kPlanes * CW;
  static constexpr int kStages = 4;
};

// One plane's copies: where the segment lies in the plane at level 1, where
// it goes in a stage, and its bytes (0: this lane copies nothing).
template <class R>
struct PlaneCopy {
  const R *src;
  int dst;
  unsigned bytes;
};

// whether x holds for some thread of the block, a block barrier
template <int CW>
__device__ __forceinline__ bool block_any(bool x) {
  if constexpr (CW == 32) {
    x = __any_sync(0xffffffffu, x);
    __syncwarp();
    return x;
  } else {
    return __syncthreads_or(x);
  }
}
template <int CW>
__device__ __forceinline__ void block_sync() {
  if constexpr (CW == 32) __syncwarp();
  else __syncthreads();
}

// The FP64 form: the arithmetic of k_solve_cols_d, 31 FP64 instructions a
// column and level.
template <class R, int CW>
__global__ void __launch_bounds__(CW, CW == 32 ? 24 : 768 / CW) k_solve_stream_d(const Dom<R> *__restrict__ doms,
    int advoff, int last, const WorkItem *__restrict__ wl) {
  grid_begin();
  static_assert(sizeof(R) == sizeof(double), "FP64 member");
  using Sh = SolveShape<R, CW>;
  constexpr int NS = Sh::kStages, ZW = Sh::kZW;
  extern __shared__ __align__(16) double dv_smem[];
  __shared__ __align__(8) uint64_t mbar[NS];
  const WorkItem wi = wl ? wl[blockIdx.x]
                          : WorkItem{(int16_t)blockIdx.z, (int16_t)blockIdx.x, (int16_t)blockIdx.y, 0};
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const int t = (int)threadIdx.x;
  const int x0 = (int)wi.a * CW;
  const int i = (int)wi.b + 2;
  if (x0 + 1 > g.jx - 2 || i > g.iy - 2) return;  // uniform over the block
  const int j = x0 + t + 1;
  const bool act = j >= 2 && j <= g.jx - 2;
  const int kz = g.kz;
  const Scal &c = D.c;
  const Stat<R> &sa = D.sa;
  const int adv = (D.clk->adv_role + advoff) & 1;
  const int PS = (int)g.PS, P = g.P;
  const size_t r0 = g.at2(1, i);
  const SoundScratch<R> ss = sound_scratch(D);
  const double *__restrict__ zraw = D.zdiv2 + r0;
  double *__restrict__ s = D.s + r0;
  double *__restrict__ w = D.w + r0;
  double *__restrict__ pai = D.pai[adv] + r0;
  double *__restrict__ zp = D.tetavf + r0;
  double *__restrict__ zfs = ss.zf + r0;
  double *__restrict__ mul = ss.mul + r0;
  const double gdts = kGrav * c.dtsound;
  const int ij_off = j - 1;
  const bool filt = c.divfilter != 0;
  const int xe = min(x0 + CW, P);
  const int zs = x0 >= Sh::kHalo ? x0 - Sh::kHalo : 0, ze = min(x0 + CW + Sh::kHalo, P);
  const unsigned wb = (unsigned)(xe - x0) * 8u, zb = (unsigned)(ze - zs) * 8u;
  const int zc = x0 + t - zs;
  auto stage = [&](int b) { return dv_smem + (size_t)b * Sh::kStage; };
  constexpr int F0 = 3 * ZW;  // the first plane's offset
  const int nd = kz - 1, nu = kz;
  // this lane's plane of the downward pass (level m: divergence, s, the
  // vertical divergence factor, pai, b; interface m+1: w, Z, G)
  PlaneCopy<R> pc{nullptr, 0, 0u};
  unsigned dn_bytes = (filt ? 3u : 1u) * zb + 7u * wb;
  if (t < 32) {
    switch (t) {
      case 0: pc = {zraw + zs, 0, zb}; break;
      case 1: pc = {zraw - P + zs, ZW, filt ? zb : 0u}; break;
      case 2: pc = {zraw + P + zs, 2 * ZW, filt ? zb : 0u}; break;
      case 3: pc = {s + x0, F0, wb}; break;
      case 4: pc = {sa.sv_a + r0 + x0, F0 + CW, wb}; break;
      case 5: pc = {pai + x0, F0 + 2 * CW, wb}; break;
      case 6: pc = {sa.sv_b + r0 + x0, F0 + 3 * CW, wb}; break;
      case 7: pc = {w + PS + x0, F0 + 4 * CW, wb}; break;
      case 8: pc = {zp + PS + x0, F0 + 5 * CW, wb}; break;
      case 9: pc = {ss.g + r0 + PS + x0, F0 + 6 * CW, wb}; break;
      default: break;
    }
  }
  // warp 0: the copies of down unit u (m = kz-1-u) or up unit v (m = v+2)
  auto issue_down = [&](int u, int b) {
    fence_proxy_async();
    if (t == 0) {
      mbar_expect_tx(&mbar[b], dn_bytes);
    }
    __syncwarp();
    if (pc.bytes) bulk_load(stage(b) + pc.dst, pc.src + (kz - 2 - u) * PS, pc.bytes, &mbar[b]);
  };
  auto issue_up = [&](int v, int b) {
    const bool top = v == kz - 1;
    fence_proxy_async();
    if (t == 0) {
      mbar_expect_tx(&mbar[b], ((last ? 7u : 5u) - (top ? 1u : 0u)) * wb);
    }
    __syncwarp();
    if (pc.bytes && !(top && t == 1)) bulk_load(stage(b) + pc.dst, pc.src + v * PS, pc.bytes, &mbar[b]);
  };
  auto bail = [&](int gnext, int gend) {
    if (t == 0) {
      atomicOr(&D.clk->fault, 1);
      for (int q = gnext; q < gend && q < gnext + NS; ++q) mbar_wait_bounded(&mbar[q % NS], (unsigned)((q / NS) & 1));
    }
  };
  if (t == 0) {
    for (int q = 0; q < NS; ++q) mbar_init(&mbar[q], 1);
    fence_mbar_init();
  }
  block_sync<CW>();
  if (t < 32)
    for (int u = 0; u < NS && u < nd; ++u) issue_down(u, u);
  // carried from the level below
  LevelD vk{};
  double wnext = 0.0, wkp1 = 0.0;
  if (act) {
    const int o = (kz - 1) * PS + ij_off;
    vk.s = s[o];
    vk.pai = pai[o];
    const double ds = vk.s - s[kz * PS + ij_off];
    if (filt)
      level_d(vk, true, sa.xknu[kz - 1], zraw[o], zraw[o - 1], zraw[o + 1], zraw[o - P], zraw[o + P],
              sa.sv_a[r0 + o], ds, sa.sv_b[r0 + o]);
    else
      level_d(vk, false, 0.0, zraw[o], 0.0, 0.0, 0.0, 0.0, sa.sv_a[r0 + o], ds, sa.sv_b[r0 + o]);
    wnext = w[kz * PS + ij_off];  // w(kz+1) = -s(kz+1)
  }
  for (int u = 0; u < nd; ++u) {
    const int k = kz - u, m = k - 1;
    const int b = u % NS;
    const bool landed = mbar_wait_bounded(&mbar[b], (unsigned)((u / NS) & 1));
    const double *st = stage(b);
    if (act) {
      const int o = (k - 1) * PS + ij_off;
      const double *f0 = st + F0 + t;
      LevelD vm;
      vm.s = f0[0];
      vm.pai = f0[2 * CW];
      const double wold = f0[4 * CW];
      if (filt)
        level_d(vm, true, sa.xknu[m - 1], st[zc], st[zc - 1], st[zc + 1], st[ZW + zc], st[2 * ZW + zc], f0[CW],
                vm.s - vk.s, f0[3 * CW]);
      else
        level_d(vm, false, 0.0, st[zc], 0.0, 0.0, 0.0, 0.0, f0[CW], vm.s - vk.s, f0[3 * CW]);
      const double Z = __fma_rn(-wold, f0[6 * CW], f0[5 * CW]);
      zfs[o] = vk.zf;
      zp[o] = Z;
      eliminate_d(wnext, wkp1, coef_d(vm, vk, Z, wold, sa.ffilt[k - 1], gdts));
      w[o] = wnext;
      mul[o] = wkp1;
      vk = vm;
    }
    if (block_any<CW>(!landed)) {
      bail(u + 1, min(nd, u + NS));  // the units issued and not read
      return;
    }
    // stage b is read: refill it
    if (t < 32 && u + NS < nd) issue_down(u + NS, b);
  }
  if (act) zfs[ij_off] = vk.zf;  // level 1
  if (t < 32) {
    pc = {nullptr, 0, 0u};
    // this lane's plane of the upward pass (level m-1: pai, divergence, dtrdz*fmz and,
    // after the last substep, s and fmzf; interface m: w, multiplier)
    switch (t) {
      case 0: pc = {w + PS + x0, F0, wb}; break;
      case 1: pc = {mul + PS + x0, F0 + CW, wb}; break;  // not at m = kz+1
      case 2: pc = {pai + x0, F0 + 2 * CW, wb}; break;
      case 3: pc = {zfs + x0, F0 + 3 * CW, wb}; break;
      case 4: pc = {sa.sv_c + r0 + x0, F0 + 4 * CW, wb}; break;
      case 5: pc = {s + x0, F0 + 5 * CW, last ? wb : 0u}; break;
      case 6: pc = {sa.fmzf_d + r0 + x0, F0 + 6 * CW, last ? wb : 0u}; break;
      default: break;
    }
  }
  fence_proxy_async_global();
  block_sync<CW>();
  if (t < 32)
    for (int v = 0; v < NS && v < nu; ++v) issue_up(v, (nd + v) % NS);
  // Exner (:668-671) of level k-1 once w(k) is known, and s (:728-734)
  double wprev = act ? w[ij_off] : 0.0;  // w(1) = 0
  for (int v = 0; v < nu; ++v) {
    const int k = v + 2, gu = nd + v;
    const int b = gu % NS;
    const bool landed = mbar_wait_bounded(&mbar[b], (unsigned)((gu / NS) & 1));
    if (act) {
      const double *f0 = stage(b) + F0 + t;
      const int o = v * PS + ij_off;
      double wk = f0[0];
      if (k <= kz) {
        wk = __fma_rn(f0[CW], wprev, wk);
        w[o + PS] = wk;
      }
      pai[o] = exner_d(f0[2 * CW], f0[3 * CW], f0[4 * CW], wprev, wk);
      if (last && k >= 3) s[o] = (wprev + f0[5 * CW]) * f0[6 * CW];
      wprev = wk;
    }
    if (block_any<CW>(!landed)) {
      bail(gu + 1, nd + min(nu, v + NS));
      return;
    }
    if (t < 32 && v + NS < nu) issue_up(v + NS, b);
  }
  if (last && act) {
    s[ij_off] = 0.0;
    s[kz * PS + ij_off] = 0.0;
  }
}

// The mixed form: the arithmetic of k_solve_cols_f.
// Seven blocks an SM (64 registers): 793 us of four solves at 512x512x41; six
// 804, eight (56 registers) 817, five 893.
template <class R, int CW, bool DFR>
__global__ void __launch_bounds__(CW, 7) k_solve_stream_f(const Dom<R> *__restrict__ doms,
    int advoff, int last, const WorkItem *__restrict__ wl) {
  grid_begin();
  static_assert(sizeof(R) == sizeof(float), "FP32 fields");
  using Sh = SolveShape<R, CW>;
  constexpr int NS = Sh::kStages, ZW = Sh::kZW;
  extern __shared__ __align__(16) float sv_smem[];
  __shared__ __align__(8) uint64_t mbar[NS];
  const WorkItem wi = wl ? wl[blockIdx.x]
                          : WorkItem{(int16_t)blockIdx.z, (int16_t)blockIdx.x, (int16_t)blockIdx.y, 0};
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const int t = (int)threadIdx.x;
  const int x0 = (int)wi.a * CW;            // first column (0-based j-1) of the block
  const int i = (int)wi.b + 2;
  if (x0 + 1 > g.jx - 2 || i > g.iy - 2) return;  // uniform over the block
  const int j = x0 + t + 1;
  const bool act = j >= 2 && j <= g.jx - 2;
  const int kz = g.kz;
  const Scal &c = D.c;
  const Stat<R> &sa = D.sa;
  const int adv = (D.clk->adv_role + advoff) & 1;
  const size_t F = g.field3(), F1 = g.PS * (size_t)(kz + 1);
  const int PS = (int)g.PS, P = g.P;
  const size_t r0 = g.at2(1, i);                  // row i, column 1
  const SoundScratch<R> ss = sound_scratch(D);
  // row bases (column 1 of row i, level 1)
  float *__restrict__ pai_h = reinterpret_cast<float *>(D.pai[adv]) + r0;
  float *__restrict__ pai_l = pai_h + F;
  float *__restrict__ z_h = reinterpret_cast<float *>(D.tetavf) + r0;
  float *__restrict__ z_l = z_h + F1;
  float *__restrict__ zfs = ss.zf + r0;
  float *__restrict__ mul = ss.mul + r0;
  float *__restrict__ w_lo = ss.w_lo + r0;
  float *__restrict__ mul_lo = ss.mul_lo + r0;
  const float *__restrict__ zraw = D.zdiv2 + r0;
  const float *__restrict__ fmz = sa.fmz + r0;
  float *__restrict__ s = D.s + r0;
  float *__restrict__ w = D.w + r0;
  const float dtrdz = c.dtsoundf * c.rdzitaf;
  const F2 ngdts{-c.gdts_hi, -c.gdts_lo};
  const int ij_off = j - 1;                       // this thread's column offset in a row
  const int32_t ib = act ? sa.ibnd_cr[r0 + ij_off] : 0;
  const int nsp = c.nspgx;
  const bool filt = c.divfilter != 0;
  // copy extents: the block's columns, and the raw divergence with its halo
  const int xe = min(x0 + CW, P);
  const int zs = x0 >= Sh::kHalo ? x0 - Sh::kHalo : 0, ze = min(x0 + CW + Sh::kHalo, P);
  const unsigned wb = (unsigned)(xe - x0) * 4u, zb = (unsigned)(ze - zs) * 4u;
  const int zc = x0 + t - zs;                     // this column in a halo row
  auto stage = [&](int b) { return sv_smem + (size_t)b * Sh::kStage; };
  constexpr int F0 = 3 * ZW;
  const int nd = kz - 1, nu = kz;                 // down units: m = kz-1 .. 1, up units: m = 2 .. kz+1
  PlaneCopy<R> pc{nullptr, 0, 0u};
  const unsigned dn_bytes = (filt ? 3u : 1u) * zb + 8u * wb;
  if (t < 32) {
    switch (t) {
      case 0: pc = {zraw + zs, 0, zb}; break;
      case 1: pc = {zraw - P + zs, ZW, filt ? zb : 0u}; break;
      case 2: pc = {zraw + P + zs, 2 * ZW, filt ? zb : 0u}; break;
      case 3: pc = {s + x0, F0, wb}; break;
      case 4: pc = {fmz + x0, F0 + CW, wb}; break;
      case 5: pc = {pai_h + x0, F0 + 2 * CW, wb}; break;
      case 6: pc = {pai_l + x0, F0 + 3 * CW, wb}; break;
      case 7: pc = {w + PS + x0, F0 + 4 * CW, wb}; break;
      case 8: pc = {ss.g + r0 + PS + x0, F0 + 5 * CW, wb}; break;
      case 9: pc = {z_h + PS + x0, F0 + 6 * CW, wb}; break;
      case 10: pc = {z_l + PS + x0, F0 + 7 * CW, wb}; break;
      default: break;
    }
  }
  auto issue_down = [&](int u, int b) {
    fence_proxy_async();
    if (t == 0) {
      mbar_expect_tx(&mbar[b], dn_bytes);
    }
    __syncwarp();
    if (pc.bytes) bulk_load(stage(b) + pc.dst, pc.src + (kz - 2 - u) * PS, pc.bytes, &mbar[b]);
  };
  auto issue_up = [&](int v, int b) {
    const bool top = v == kz - 1;
    fence_proxy_async();
    if (t == 0) {
      mbar_expect_tx(&mbar[b], (5u + (last ? 2u : 0u) + (top ? 0u : DFR ? 3u : 1u)) * wb);
    }
    __syncwarp();
    if (pc.bytes && !(top && t >= 1 && t <= 3))
      bulk_load(stage(b) + pc.dst, pc.src + v * PS, pc.bytes, &mbar[b]);
  };
  // a failed wait (a copy that never landed): record it, let the copies in
  // flight land (bounded) and leave
  auto bail = [&](int gnext, int gend) {
    if (t == 0) {
      atomicOr(&D.clk->fault, 1);
      for (int q = gnext; q < gend && q < gnext + NS; ++q) mbar_wait_bounded(&mbar[q % NS], (unsigned)((q / NS) & 1));
    }
  };
  if (t == 0) {
    for (int q = 0; q < NS; ++q) mbar_init(&mbar[q], 1);
    fence_mbar_init();
  }
  block_sync<CW>();
  if (t < 32)
    for (int u = 0; u < NS && u < nd; ++u) issue_down(u, u);

  auto bweight = [&](int m) {
    return ib > 0 ? 1.f - sa.hefc_r[(size_t)(ib - 1) + (size_t)(m - 1) * nsp] : 1.f;
  };
  // level kz and the interface below it straight from memory (once)
  LevelF vk{};
  F2 wnext{0.f, 0.f}, wkp1{0.f, 0.f};
  if (act) {
    const int o = (kz - 1) * PS + ij_off;
    vk.s = s[o];
    vk.pai = F2{pai_h[o], pai_l[o]};
    const float fz = __fmul_rn(dtrdz, fmz[o]), ds = vk.s - s[kz * PS + ij_off];
    if (filt)
      level_f(vk, true, sa.xknu_r[kz - 1], zraw[o], zraw[o - 1], zraw[o + 1], zraw[o - P], zraw[o + P], bweight(kz),
              fz, ds);
    else
      level_f(vk, false, 0.f, zraw[o], 0.f, 0.f, 0.f, 0.f, bweight(kz), fz, ds);
    wnext.hi = w[kz * PS + ij_off];
  }
  for (int u = 0; u < nd; ++u) {
    const int k = kz - u, m = k - 1;
    const int b = u % NS;
    const bool landed = mbar_wait_bounded(&mbar[b], (unsigned)((u / NS) & 1));
    const float *st = stage(b);
    if (act) {
      const int o = (k - 1) * PS + ij_off;
      const float *f0 = st + F0 + t;
      LevelF vm;
      vm.s = f0[0];
      vm.pai = F2{f0[2 * CW], f0[3 * CW]};
      const float fz = __fmul_rn(dtrdz, f0[CW]), wold = f0[4 * CW];
      if (filt)
        level_f(vm, true, sa.xknu_r[m - 1], st[zc], st[zc - 1], st[zc + 1], st[ZW + zc], st[2 * ZW + zc], bweight(m),
                fz, vm.s - vk.s);
      else
        level_f(vm, false, 0.f, st[zc], 0.f, 0.f, 0.f, 0.f, bweight(m), fz, vm.s - vk.s);
      zfs[o] = vk.zf;
      const F2 Z = df_add_f(F2{f0[6 * CW], f0[7 * CW]}, -__fmul_rn(wold, f0[5 * CW]));
      z_h[o] = Z.hi;
      z_l[o] = Z.lo;
      eliminate_f<DFR>(wnext, wkp1, coef_f(vm, vk, Z, wold, sa.ffilt_r[k - 1], ngdts));
      w[o] = wnext.hi;
      mul[o] = wkp1.hi;
      if constexpr (DFR) {
        w_lo[o] = wnext.lo;
        mul_lo[o] = wkp1.lo;
      }
      vk = vm;
    }
    if (block_any<CW>(!landed)) {
      bail(u + 1, min(nd, u + NS));  // the units issued and not read
      return;
    }
    // stage b is read: refill it
    if (t < 32 && u + NS < nd) issue_down(u + NS, b);
  }
  if (act) zfs[ij_off] = vk.zf;  // level 1
  // this thread's stores of w, mul and zfs are read back by the copy engine
  if (t < 32) {
    pc = {nullptr, 0, 0u};
    // s and fmzf (after the last substep) go where the divergence rows lay
    switch (t) {
      case 0: pc = {w + PS + x0, F0, wb}; break;
      case 1: pc = {mul + PS + x0, F0 + CW, wb}; break;             // these three
      case 2: pc = {w_lo + PS + x0, F0 + 2 * CW, DFR ? wb : 0u}; break;    // not at
      case 3: pc = {mul_lo + PS + x0, F0 + 3 * CW, DFR ? wb : 0u}; break;  // m = kz+1
      case 4: pc = {pai_h + x0, F0 + 4 * CW, wb}; break;
      case 5: pc = {pai_l + x0, F0 + 5 * CW, wb}; break;
      case 6: pc = {zfs + x0, F0 + 6 * CW, wb}; break;
      case 7: pc = {fmz + x0, F0 + 7 * CW, wb}; break;
      case 8: pc = {s + x0, 0, last ? wb : 0u}; break;
      case 9: pc = {sa.fmzf + r0 + x0, ZW, last ? wb : 0u}; break;
      default: break;
    }
  }
  fence_proxy_async_global();
  block_sync<CW>();
  if (t < 32)
    for (int v = 0; v < NS && v < nu; ++v) issue_up(v, (nd + v) % NS);
  F2 wprev{act ? w[ij_off] : 0.f, 0.f};  // w(1) = 0
  for (int v = 0; v < nu; ++v) {
    const int k = v + 2, gu = nd + v;
    const int b = gu % NS;
    const bool landed = mbar_wait_bounded(&mbar[b], (unsigned)((gu / NS) & 1));
    if (act) {
      const float *st = stage(b);
      const float *f0 = st + F0 + t;
      const int o = v * PS + ij_off;
      F2 wk{f0[0], 0.f};
      if (k <= kz) {
        if constexpr (DFR) wk = back_f<DFR>(F2{wk.hi, f0[2 * CW]}, F2{f0[CW], f0[3 * CW]}, wprev);
        else wk = back_f<DFR>(wk, F2{f0[CW], 0.f}, wprev);
        w[o + PS] = df_f(wk);
      }
      // Exner of level k-1 (and s after the last substep)
      const F2 pn = exner_f(F2{f0[4 * CW], f0[5 * CW]}, f0[6 * CW], __fmul_rn(dtrdz, f0[7 * CW]), wprev, wk);
      pai_h[o] = pn.hi;
      pai_l[o] = pn.lo;
      if (last && k >= 3) s[o] = (df_f(wprev) + st[t]) * st[ZW + t];
      wprev = wk;
    }
    if (block_any<CW>(!landed)) {
      bail(gu + 1, nd + min(nu, v + NS));
      return;
    }
    if (t < 32 && v + NS < nu) issue_up(v + NS, b);
  }
  if (last && act) {
    s[ij_off] = 0.f;
    s[kz * PS + ij_off] = 0.f;
  }
}

// Main/mod_moloch.F90:677-721 with divergence_damping :738-765 folded in, FP64
template <class R, int LV>
__global__ void k_sound_momentum(const Dom<R> *__restrict__ doms, int uvoff, int advoff,
                                 int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  const WorkItem wi = work_item(wl, tiles_j);
  static_assert(sizeof(R) == sizeof(double), "FP64 member");
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const Scal &c = D.c;
  const Stat<R> &sa = D.sa;
  const int uv = (D.clk->uv_role + uvoff) & 1;
  const int adv = (D.clk->adv_role + advoff) & 1;
  const R *__restrict__ u_in = D.u[uv];
  const R *__restrict__ v_in = D.v[uv];
  R *__restrict__ u_out = D.u[uv ^ 1];
  R *__restrict__ v_out = D.v[uv ^ 1];
  const R *__restrict__ zraw = D.zdiv2;
  const double *__restrict__ pai = D.pai[adv];
  const SoundScratch<R> ss = sound_scratch(D);
  const Pt q = point_at<LV>(wi, 1, 1);
  const int j = q.j, i = q.i;
  if (j > g.jx || i > g.iy || q.k > g.kz) return;
  const size_t ij = g.at2(j, i);
  const size_t PS = g.PS;
  const bool has_u = i <= g.iy - 1;
  const bool has_v = j <= g.jx - 1;
  const bool upd_u = has_u && j >= 2 && j <= g.jx - 1 && i >= 2 && i <= g.iy - 2;
  const bool upd_v = has_v && j >= 2 && j <= g.jx - 2 && i >= 2 && i <= g.iy - 1;
  const double cor_u = upd_u ? sa.mo_cu[ij] : 0.0, cor_v = upd_v ? sa.mo_cv[ij] : 0.0;
  const size_t W = 1, S = (size_t)g.P;
  // Six FP64 instructions a wind point (the pipe that bounds this kernel):
  // the constant products dxrdt*xkdamp*msfu, g*dts*hx*gzitakh and coru*dts
  // come from bind time, zcx*cp/2*(theta_v sum) from sound_prep.
#pragma unroll
  for (int k = q.k; k < q.k + LV && k <= g.kz; ++k) {
    const size_t o = ij + (size_t)(k - 1) * PS;
    if (has_u) {
      double un = u_in[o];
      if (upd_u) {
        if (c.divdamp) un = __fma_rn(sa.mo_du[o], zraw[o] - zraw[o - W], un);
        const double r = __fma_rn(-ss.cu[o], pai[o] - pai[o - W], __fma_rn(cor_u, v_in[o], -sa.mo_gu[o]));
        un = __fma_rn(relax_weight(sa.ibnd_ud, sa.hefc, c.nspgx, ij, k), r, un);
      }
      u_out[o] = un;
    }
    if (has_v) {
      double vn = v_in[o];
      if (upd_v) {
        if (c.divdamp) vn = __fma_rn(sa.mo_dv[o], zraw[o] - zraw[o - S], vn);
        const double r = __fma_rn(-ss.cv[o], pai[o] - pai[o - S], __fma_rn(-cor_v, u_in[o], -sa.mo_gv[o]));
        vn = __fma_rn(relax_weight(sa.ibnd_vd, sa.hefc, c.nspgx, ij, k), r, vn);
      }
      v_out[o] = vn;
    }
  }
}

// 16 bytes at p (16-byte aligned) as 4 floats / 4 ints
__device__ __forceinline__ void ld4(float (&x)[4], const float *p) {
  const float4 v = *reinterpret_cast<const float4 *>(p);
  x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
__device__ __forceinline__ void ld4i(int (&x)[4], const int32_t *p) {
  const int4 v = *reinterpret_cast<const int4 *>(p);
  x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
// x[q] at q = -1..3: the lane's own elements, the one west of them read singly
struct West4 {
  float w, x[4];
  __device__ __forceinline__ float at(int q) const { return q < 0 ? w : x[q]; }
};

// Blocks of 128 threads an SM the four-column point kernels are compiled for
// (the register budget follows).  Momentum, four levels a thread: 5 blocks (96
// registers, a few spilled to L1) 0.377 ms a moist 512x512x41 step, against
// 0.385 at 4 and 0.409 at 6; one level a thread, where few blocks run anyway:
// 4 blocks (no spills) 0.215 ms a rotated 150x187x40 step, 0.223 at 5.  The
// divergence: 4 blocks with two levels' loads in flight 0.274 ms (one level's
// 0.330), 5 blocks 0.300, 3 blocks 0.323.
template <int LV>
constexpr int momentum_blocks() {
  return LV == 1 ? 4 : 5;
}

// The divergence and s of a mixed member (the same equations as
// k_sound_div) with lanes of four consecutive columns: 16-byte loads at the
// lane's points and the row north of them, the east neighbour of the last
// element read singly, the level below carried from the previous level.
template <class R, int LV>
__global__ void __launch_bounds__(128, 4) k_sound_div_v4(const Dom<R> *__restrict__ doms, int uvoff,
                                                      int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  static_assert(sizeof(R) == sizeof(float), "FP32 fields");
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const int jx = g.jx, iy = g.iy, kz = g.kz;
  const int bj = wi.a, bi = wi.b;
  const int e0 = (bj * 32 + (int)threadIdx.x) * 4;
  const int i = bi * (int)blockDim.y + (int)threadIdx.y + 1;
  const int k0 = (int)wi.c * LV + 1;
  if (e0 + 1 > jx - 1 || i > iy - 1 || k0 > kz) return;
  const Scal &c = D.c;
  const Stat<R> &sa = D.sa;
  const int uv = (D.clk->uv_role + uvoff) & 1;
  const float *__restrict__ u = D.u[uv];
  const float *__restrict__ v = D.v[uv];
  float *__restrict__ zdiv2 = D.zdiv2;
  float *__restrict__ sv = D.s;
  float *__restrict__ w = D.w;
  const unsigned P = (unsigned)g.P, PS = (unsigned)g.PS;
  const unsigned ij = (unsigned)e0 + (unsigned)(i - 1) * P;
  const bool east = e0 + 4 <= jx - 1;  // element 3 has an east neighbour to read
  bool has[4], inner[4];
  bool all = true;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int j = e0 + q + 1;
    has[q] = j <= jx - 1;
    inner[q] = j >= 2 && j <= jx - 2 && i >= 2 && i <= iy - 2;
    all = all && has[q];
  }
  const bool any_inner = inner[0] || inner[1] || inner[2] || inner[3];
  auto next4 = [&](float (&e)[4], const float (&x)[4], const float *arr, unsigned o) {
    e[0] = x[1]; e[1] = x[2]; e[2] = x[3];
    e[3] = east ? arr[o + 4] : 0.f;
  };
  float rmu0[4], rmu1[4], rmv0[4], rmv1[4], mfac[4], hx0[4], hx1[4], hy0[4], hy1[4];
  ld4(rmu0, sa.rmu + ij);
  next4(rmu1, rmu0, sa.rmu, ij);
  ld4(rmv0, sa.rmv + ij);
  ld4(rmv1, sa.rmv + ij + P);
  ld4(mfac, (c.lrotllr ? sa.msfx : sa.mx2) + ij);
  ld4(hx0, sa.hx + ij);
  next4(hx1, hx0, sa.hx, ij);
  ld4(hy0, sa.hy + ij);
  ld4(hy1, sa.hy + ij + P);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (!inner[q]) hx0[q] = hx1[q] = hy0[q] = hy1[q] = 0.f;
    // the face fluxes' 2-D factors dts/dx/m (rotated: dts/dx for u)
    rmu0[q] = c.lrotllr ? c.dtrdxsf : mul_r(c.dtrdxsf, rmu0[q]);
    rmu1[q] = c.lrotllr ? c.dtrdxsf : mul_r(c.dtrdxsf, rmu1[q]);
    rmv0[q] = mul_r(c.dtrdxsf, rmv0[q]);
    rmv1[q] = mul_r(c.dtrdxsf, rmv1[q]);
  }
  // the winds of the level below (for s)
  float um[4], upm[4], vm[4], vpm[4];
  if (k0 >= 2 && any_inner) {
    const unsigned om = ij + (unsigned)(k0 - 2) * PS;
    ld4(um, u + om);
    next4(upm, um, u, om);
    ld4(vm, v + om);
    ld4(vpm, v + om + P);
  }
#pragma unroll 2
  for (int k = k0; k < k0 + LV && k <= kz; ++k) {
    const unsigned o = ij + (unsigned)(k - 1) * PS;
    float u0[4], u1[4], v0[4], v1[4], fu0[4], fu1[4], fv0[4], fv1[4], fz[4], zd[4];
    ld4(u0, u + o);
    next4(u1, u0, u, o);
    ld4(v0, v + o);
    ld4(v1, v + o + P);
    ld4(fu0, sa.rfmzu + o);
    next4(fu1, fu0, sa.rfmzu, o);
    ld4(fv0, sa.rfmzv + o);
    ld4(fv1, sa.rfmzv + o + P);
    ld4(fz, sa.fmz + o);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      zd[q] = divergence<float>(mul_r(fz[q], mfac[q]), u0[q], mul_r(fu0[q], rmu0[q]), u1[q], mul_r(fu1[q], rmu1[q]),
                                v0[q], mul_r(fv0[q], rmv0[q]), v1[q], mul_r(fv1[q], rmv1[q]));
    if (all) {
      *reinterpret_cast<float4 *>(zdiv2 + o) = make_float4(zd[0], zd[1], zd[2], zd[3]);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (has[q]) zdiv2[o + q] = zd[q];
    }
    if (any_inner) {
      if (k >= 2) {
        const float gk = sa.gzitak_r[k - 1];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (inner[q])
            sv[o + q] = mul_r(slope_wind<float>(u0[q] + um[q], hx0[q], u1[q] + upm[q], hx1[q], v0[q] + vm[q], hy0[q],
                                                v1[q] + vpm[q], hy1[q]),
                              gk);
      }
      if (k == kz) {
        const unsigned ot = ij + (unsigned)kz * PS;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (inner[q]) {
            const float skp1 = -0.5f * slope_wind<float>(u0[q], hx0[q], u1[q], hx1[q], v0[q], hy0[q], v1[q], hy1[q]);
            sv[ot + q] = skp1;
            w[ot + q] = -skp1;
          }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        um[q] = u0[q]; upm[q] = u1[q]; vm[q] = v0[q]; vpm[q] = v1[q];
      }
    }
  }
}

// The momentum update of a mixed member (the same equations as
// k_sound_momentum) with lanes of four consecutive columns: 16-byte loads of
// every field at the lane's points and the row south of them; the west
// neighbours are the lane's own elements but for the first, read singly.  A
// block is 32 lanes x 4 rows; grid x = 128-column tiles times row tiles, y =
// level chunks, z = member.
template <class R, int LV>
__global__ void __launch_bounds__(128, momentum_blocks<LV>()) k_sound_momentum_v4(const Dom<R> *__restrict__ doms,
                                                           int uvoff, int advoff, int tiles_j,
    const WorkItem *__restrict__ wl) {
  if constexpr (LV == 1) grid_begin();
  static_assert(sizeof(R) == sizeof(float), "FP32 fields");
  const WorkItem wi = work_item(wl, tiles_j);
  const Dom<R> &D = doms[wi.m];
  if (!D.active) return;
  const Geom g = D.g;
  const int jx = g.jx, iy = g.iy, kz = g.kz;
  const int bj = wi.a, bi = wi.b;
  const int e0 = (bj * 32 + (int)threadIdx.x) * 4;  // j-1 of the lane's first column
  const int i = bi * (int)blockDim.y + (int)threadIdx.y + 1;
  const int k0 = (int)wi.c * LV + 1;
  if (e0 + 1 > jx || i > iy || k0 > kz) return;
  const Scal &c = D.c;
  const Stat<R> &sa = D.sa;
  const int uv = (D.clk->uv_role + uvoff) & 1;
  const int adv = (D.clk->adv_role + advoff) & 1;
  const float *__restrict__ u_in = D.u[uv];
  const float *__restrict__ v_in = D.v[uv];
  float *__restrict__ u_out = D.u[uv ^ 1];
  float *__restrict__ v_out = D.v[uv ^ 1];
  const float *__restrict__ zraw = D.zdiv2;
  const size_t F = g.field3();
  const float *__restrict__ th_h = reinterpret_cast<const float *>(D.tetav[adv]);
  const float *__restrict__ th_l = th_h + F;
  const float *__restrict__ pa_h = reinterpret_cast<const float *>(D.pai[adv]);
  const float *__restrict__ pa_l = pa_h + F;
  const float dts = c.dtsoundf, dtrdx = c.dtrdxsf, dxrdt = c.dxrdtf;
  const float zfz = float(kGrav) * dts;
  const float halfcp = 0.5f * float(kCpd);
  const unsigned P = (unsigned)g.P;
  const unsigned ij = (unsigned)e0 + (unsigned)(i - 1) * P;
  const bool west = e0 >= 1, south = i >= 2;
  bool upd_u[4], upd_v[4], has_u[4], has_v[4];
  bool all_u = true, all_v = true;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int j = e0 + q + 1;
    has_u[q] = i <= iy - 1 && j <= jx;
    has_v[q] = j <= jx - 1;
    upd_u[q] = j >= 2 && j <= jx - 1 && i >= 2 && i <= iy - 2;
    upd_v[q] = j >= 2 && j <= jx - 2 && i >= 2 && i <= iy - 1;
    all_u = all_u && has_u[q];
    all_v = all_v && has_v[q];
  }
  // 2-D coefficients of the lane's columns (zero where nothing is updated)
  float mu[4], hx4[4], cu4[4], mv[4], hy4[4], cv4[4];
  int ibu[4], ibv[4];
  ld4(mu, sa.msfu + ij);
  ld4(hx4, sa.hx + ij);
  ld4(cu4, sa.coru + ij);
  ld4(mv, sa.msfv + ij);
  ld4(hy4, sa.hy + ij);
  ld4(cv4, sa.corv + ij);
  ld4i(ibu, sa.ibnd_ud + ij);
  ld4i(ibv, sa.ibnd_vd + ij);
  const int nsp = c.nspgx;
  // the columns' factors coru*dts and g*dts*hx, and v's; 1 for msfv of the
  // rotated pole
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    cu4[q] = mul_r(cu4[q], dts);
    hx4[q] = mul_r(zfz, hx4[q]);
    cv4[q] = mul_r(cv4[q], dts);
    hy4[q] = mul_r(zfz, hy4[q]);
    if (c.lrotllr) mv[q] = 1.f;
  }
  const float kpg = mul_r(dtrdx, halfcp);
  for (int k = k0; k < k0 + LV && k <= kz; ++k) {
    const unsigned o = ij + (unsigned)(k - 1) * (unsigned)g.PS;
    float un[4], vn[4], uo[4], vo[4];
    ld4(uo, u_in + o);
    ld4(vo, v_in + o);
    West4 zr, th, tl, ph, pl;
    ld4(zr.x, zraw + o);
    ld4(th.x, th_h + o);
    ld4(tl.x, th_l + o);
    ld4(ph.x, pa_h + o);
    ld4(pl.x, pa_l + o);
    zr.w = th.w = tl.w = ph.w = pl.w = 0.f;
    if (west) {
      zr.w = zraw[o - 1];
      th.w = th_h[o - 1];
      tl.w = th_l[o - 1];
      ph.w = pa_h[o - 1];
      pl.w = pa_l[o - 1];
    }
    float zs[4] = {0.f, 0.f, 0.f, 0.f}, ts[4] = {0.f, 0.f, 0.f, 0.f}, tsl[4] = {0.f, 0.f, 0.f, 0.f};
    float ps[4] = {0.f, 0.f, 0.f, 0.f}, psl[4] = {0.f, 0.f, 0.f, 0.f};
    if (south) {
      ld4(zs, zraw + o - P);
      ld4(ts, th_h + o - P);
      ld4(tsl, th_l + o - P);
      ld4(ps, pa_h + o - P);
      ld4(psl, pa_l + o - P);
    }
    const float gk = sa.gzitakh_r[k - 1];
    const float xd = mul_r(dxrdt, sa.xkdamp_r[k - 1]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float a = uo[q];
      if (upd_u[q]) {
        if (c.divdamp) a = fma_r(mul_r(xd, mu[q]), zr.x[q] - zr.at(q - 1), a);
        const float kp = mul_r(mul_r(kpg, mu[q]), (th.at(q - 1) + th.x[q]) + (tl.at(q - 1) + tl.x[q]));
        const int ib = ibu[q];
        const float bw = ib > 0 ? 1.f - sa.hefc_r[(size_t)(ib - 1) + (size_t)(k - 1) * nsp] : 1.f;
        const float pd = (ph.x[q] - ph.at(q - 1)) + (pl.x[q] - pl.at(q - 1));
        a = fma_r(bw, fma_r(-kp, pd, fma_r(cu4[q], vo[q], -mul_r(hx4[q], gk))), a);
      }
      un[q] = a;
      float b = vo[q];
      if (upd_v[q]) {
        if (c.divdamp) b = fma_r(mul_r(xd, mv[q]), zr.x[q] - zs[q], b);
        const float kp = mul_r(mul_r(kpg, mv[q]), (ts[q] + th.x[q]) + (tsl[q] + tl.x[q]));
        const int ib = ibv[q];
        const float bw = ib > 0 ? 1.f - sa.hefc_r[(size_t)(ib - 1) + (size_t)(k - 1) * nsp] : 1.f;
        const float pd = (ph.x[q] - ps[q]) + (pl.x[q] - psl[q]);
        b = fma_r(bw, fma_r(-kp, pd, fma_r(-cv4[q], uo[q], -mul_r(hy4[q], gk))), b);
      }
      vn[q] = b;
    }
    if (all_u) {
      *reinterpret_cast<float4 *>(u_out + o) = make_float4(un[0], un[1], un[2], un[3]);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (has_u[q]) u_out[o + q] = un[q];
    }
    if (all_v) {
      *reinterpret_cast<float4 *>(v_out + o) = make_float4(vn[0], vn[1], vn[2], vn[3]);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (has_v[q]) v_out[o + q] = vn[q];
    }
  }
}

inline dim3 col_block(const LaunchGeom &L) { return dim3((unsigned)L.col_x, (unsigned)L.col_y); }
// grid of a point kernel over nj x ni points per level
inline dim3 pt_grid(const LaunchGeom &L, int nj, int ni, int &tiles_j) {
  tiles_j = (nj + L.col_x - 1) / L.col_x;
  if (L.wl_pt) return dim3((unsigned)L.n_pt, 1, 1);  // one block per work item
  const int ti = (ni + L.col_y - 1) / L.col_y;
  return dim3((unsigned)(tiles_j * ti), (unsigned)((L.kz + L.lv - 1) / L.lv), (unsigned)L.nmem);
}
}  // namespace

template <class R>
void Launch<R>::sound_prep(const LaunchGeom &L, const Dom<R> *d, int advoff, cudaStream_t s) {
  int tj;
  const dim3 grd = pt_grid(L, L.jx - 1, L.iy - 1, tj);
  if (L.lv == 1) step_launch(L, k_sound_prep<R, 1>, grd, col_block(L), 0, s, d, advoff, tj, L.wl_pt);
  else step_launch(L, k_sound_prep<R, 4>, grd, col_block(L), 0, s, d, advoff, tj, L.wl_pt);
}

template <class R>
void Launch<R>::sound_div(const LaunchGeom &L, const Dom<R> *d, int uvoff, cudaStream_t s) {
  if constexpr (sizeof(R) == sizeof(float)) {
    const int tj = (L.jx - 1 + 127) / 128, ti = (L.iy - 1 + 3) / 4;
    const dim3 grd = L.wl_v4 ? dim3((unsigned)L.n_v4, 1, 1)
                             : dim3((unsigned)(tj * ti), (unsigned)((L.kz + L.lv - 1) / L.lv),
                                    (unsigned)L.nmem);
    if (L.lv == 1) step_launch(L, k_sound_div_v4<R, 1>, grd, dim3(32, 4), 0, s, d, uvoff, tj, L.wl_v4);
    else step_launch(L, k_sound_div_v4<R, 4>, grd, dim3(32, 4), 0, s, d, uvoff, tj, L.wl_v4);
  } else {
    int tj;
    const dim3 grd = pt_grid(L, L.jx - 1, L.iy - 1, tj);
    if (L.lv == 1) step_launch(L, k_sound_div<R, 1>, grd, col_block(L), 0, s, d, uvoff, tj, L.wl_pt);
    else step_launch(L, k_sound_div<R, 4>, grd, col_block(L), 0, s, d, uvoff, tj, L.wl_pt);
  }
}

template <class R, int AW>
void launch_cols(const LaunchGeom &L, const Dom<R> *d, dim3 grid, int advoff, int last, cudaStream_t s) {
  const size_t smem = solve_smem(L.kz, (int)sizeof(R));
  if constexpr (sizeof(R) == sizeof(float)) {
    if (L.solve_df) step_launch(L, k_solve_cols_f<R, AW, true>, grid, solve_threads(AW), smem, s, d, advoff, last, L.wl_solve);
    else step_launch(L, k_solve_cols_f<R, AW, false>, grid, solve_threads(AW), smem, s, d, advoff, last, L.wl_solve);
  } else {
    step_launch(L, k_solve_cols_d<R, AW>, grid, solve_threads(AW), smem, s, d, advoff, last, L.wl_solve);
  }
}

template <class R>
void Launch<R>::sound_solve(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, bool last,
                            cudaStream_t s) {
  (void)uvoff;
  // (LaunchGeom's solve_x and solve_y are not used)
  constexpr int CW = solve_segment(kSolveStream, (int)sizeof(R));
  const int w = solve_segment(L.solve, (int)sizeof(R)), lst = last ? 1 : 0;
  const dim3 grid = L.wl_solve ? dim3((unsigned)L.n_solve, 1, 1)
                               : dim3((unsigned)((L.jx - 1 + w - 1) / w), (unsigned)(L.iy - 3), (unsigned)L.nmem);
  if (L.solve == kSolveCols6) {
    launch_cols<R, 6>(L, d, grid, advoff, lst, s);
  } else if (L.solve == kSolveCols3) {
    launch_cols<R, 3>(L, d, grid, advoff, lst, s);
  } else {
    using Sh = SolveShape<R, CW>;
    constexpr size_t smem = (size_t)Sh::kStages * Sh::kStage * sizeof(R);
    if constexpr (sizeof(R) == sizeof(float)) {
      if (L.solve_df) step_launch(L, k_solve_stream_f<R, CW, true>, grid, CW, smem, s, d, advoff, lst, L.wl_solve);
      else step_launch(L, k_solve_stream_f<R, CW, false>, grid, CW, smem, s, d, advoff, lst, L.wl_solve);
    } else {
      step_launch(L, k_solve_stream_d<R, CW>, grid, CW, smem, s, d, advoff, lst, L.wl_solve);
    }
  }
}

template <class R>
void Launch<R>::sound_momentum(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff,
                               cudaStream_t s) {
  if constexpr (sizeof(R) == sizeof(float)) {
    // lanes of four columns: 128 columns by 4 rows a block
    const int tj = (L.jx + 127) / 128, ti = (L.iy + 3) / 4;
    const dim3 grd = L.wl_v4 ? dim3((unsigned)L.n_v4, 1, 1)
                             : dim3((unsigned)(tj * ti), (unsigned)((L.kz + L.lv - 1) / L.lv),
                                    (unsigned)L.nmem);
    if (L.lv == 1) step_launch(L, k_sound_momentum_v4<R, 1>, grd, dim3(32, 4), 0, s, d, uvoff, advoff, tj, L.wl_v4);
    else step_launch(L, k_sound_momentum_v4<R, 4>, grd, dim3(32, 4), 0, s, d, uvoff, advoff, tj, L.wl_v4);
  } else {
    int tj;
    const dim3 grd = pt_grid(L, L.jx, L.iy, tj);
    if (L.lv == 1) step_launch(L, k_sound_momentum<R, 1>, grd, col_block(L), 0, s, d, uvoff, advoff, tj, L.wl_pt);
    else step_launch(L, k_sound_momentum<R, 4>, grd, col_block(L), 0, s, d, uvoff, advoff, tj, L.wl_pt);
  }
}

template <class R>
cudaError_t Launch<R>::configure_sound() {
  // k_solve_cols holds a column of up to kMaxLevels levels in shared memory
  const int most = (int)solve_smem(kMaxLevels, (int)sizeof(R));
  cudaError_t e = cudaSuccess;
  auto allow = [&](auto k) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  };
  if constexpr (sizeof(R) == sizeof(float)) {
    allow(k_solve_cols_f<R, 3, true>);
    allow(k_solve_cols_f<R, 3, false>);
    allow(k_solve_cols_f<R, 6, true>);
    allow(k_solve_cols_f<R, 6, false>);
  } else {
    allow(k_solve_cols_d<R, 3>);
    allow(k_solve_cols_d<R, 6>);
  }
  return e;
}

template struct Launch<double>;
template struct Launch<float>;

}  // namespace mlc
