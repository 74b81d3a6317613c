// mlc_kernels.cuh -- launch interface between the step driver and the kernels.
//
// Every kernel serves all members of a context in one launch: blockIdx.z (or
// blockIdx.y for the reduction) selects the member, whose descriptor Dom<R>
// (extents, parameters, pointers) sits in a device array.  Grids cover the
// largest member; blocks outside a smaller member's extent return at once.
// Buffer roles are read from each member's device clock plus the offsets a
// launch passes (uvoff acoustic substeps, advoff advection rounds since the
// step began), so one recorded graph replays every step.
#pragma once
#include <cuda_runtime.h>

#include "mlc_device.cuh"

namespace mlc {

// Forms of the column solves (mlc_sound.cu) and the columns of a block's row
// segment in each.
constexpr int kSolveStream = 0, kSolveCols3 = 3, kSolveCols6 = 6;
constexpr int solve_segment(int kind, int elem_bytes) {
  return kind == kSolveStream && elem_bytes == 4 ? 128 : 32;
}
// The forms with several warps a column keep kSolveArrays values a column and
// level in shared memory.
constexpr int kSolveArrays = 5;
constexpr size_t solve_smem(int kz, int elem_bytes) { return (size_t)kSolveArrays * (kz + 2) * 32 * elem_bytes; }
// Blocks of such a form resident on an SM: as many as its registers allow
// (`most`), or as the columns' levels leave room for (228 KB an SM, 1 KB and
// the barriers' 176 bytes a block beside the columns).
constexpr int solve_resident(int most, int kz, int elem_bytes) {
  const int fit = (int)(((size_t)228 << 10) / (solve_smem(kz, elem_bytes) + 1024 + 176));
  return fit < most ? fit : most;
}
// The form for `segments` 32-column row segments of columns of up to kz levels
// on 152 SMs.  A form with several warps a column takes a time for each wave of
// resident blocks, three coefficient warps 1.7 times that of six (but twice as
// many blocks fit); the streamed form takes about the same until its segments
// fill the GPU.  So the one of the two whose waves take less, and streamed once
// six warps need more than two waves (FP64; three where a block fills the SM)
// or four (mixed).  Of 220 measured cases (two precisions, 24 to 128 levels,
// 0.8 to 21 segments an SM) the form taken is within 5 % of the fastest.  us a
// launch (six | three | streamed; n segments an SM):
//          n     FP64                  mixed
//   41     1.9   37.8  45.1  85.7      19.6  27.7  65.1
//   levels 3.3   72.3  64.6  90.0      22.9  29.7  65.9
//          5.2    105   120   102      37.4  33.7  74.1
//          9.5    172   179   135      59.7  63.8  77.5
//          13.4   241   238   183      80.8  71.1  81.0
//          20.9   375   354   300       123   106   107
//   70     1.9   59.4  79.4   141      27.7  41.4   106
//          3.3    114   156   148      34.6  47.9   107
//          5.2    167   233   169      60.5  94.1   120
//          13.4   384   538   306       127   199   133
//          20.9   600   845   505       192   301   176
//   128    1.9    158   269   251      49.1  79.5   187
//          3.3    312   533   262      98.6   164   188
//          7.5    622  1073   350       202   340   223
//          13.4  1085  1872   550       357   602   237
constexpr int solve_form(long segments, int kz, int elem_bytes) {
  const bool f64 = elem_bytes == 8;
  const int r6 = solve_resident(f64 ? 2 : 4, kz, elem_bytes), r3 = solve_resident(f64 ? 5 : 8, kz, elem_bytes);
  const long w6 = (segments + 152L * r6 - 1) / (152L * r6), w3 = (segments + 152L * r3 - 1) / (152L * r3);
  const bool three = 17 * w3 < 10 * w6;
  if (f64 && three) return w3 == 1 ? kSolveCols3 : kSolveStream;
  if (w6 > (f64 ? (r6 == 1 ? 3 : 2) : 4)) return kSolveStream;
  return three ? kSolveCols3 : kSolveCols6;
}
// Tiles of end_winds: a block is kWindWarps warps, a warp a row segment of 128
// columns of which it writes kWindCols, marching over some rows.
constexpr int kWindWarps = 4, kWindCols = 120;
constexpr int wind_tiles_j(int jx) { return (jx + kWindCols - 1) / kWindCols; }
constexpr int wind_tiles_i(int iy, int rows) { return (iy + kWindWarps * rows - 1) / (kWindWarps * rows); }

// Levels of a domain, at most.
constexpr int kMaxLevels = 128;

// Extents of a launch (maxima over the members) and the launch shapes.
struct LaunchGeom {
  int jx, iy, kz, nmem;
  int col_x, col_y;      // column kernels
  int solve_x, solve_y;  // kept in the tune report; not used by the solves
  int solve;             // form of the column solves (kSolveStream ...)
  int wind_rows;         // rows of a warp of end_winds (0: FP64 members, end_uvx and end_uvstag)
  int frame_points;      // points a level of the largest member's frame (Scal::frame)
  int min_frame;         // the thinnest member's frame
  int lv;                // levels a thread of the point kernels runs (1 or 4)
  int vert_x, vert_y;    // adv_vertical
  int vert_nf;           // fields a thread of it carries (1; mixed members by size 2)
  int htile;             // adv_horizontal tile shape (hshape) asked for, -1: by size
  int size_tile, size_tile_inc;  // the shapes by size (refresh)
  int nadv_r;            // advected fields of type R per member
  int nadv_d;            // advected FP64 fields per member (mixed: theta_v, Exner)
  int red_blocks;        // reduction blocks of the largest member
  int solve_df;          // mixed solve: recurrence in double-float (1) or FP32 (0)
  // work lists of an uneven batch (device arrays; null: grids over the
  // largest member) and their lengths, one per tiling
  const WorkItem *wl_pt;     // col_x x col_y tiles, level chunks
  const WorkItem *wl_v4;     // 128 x 4 tiles, level chunks
  const WorkItem *wl_vec;    // the step end's: 16-byte lanes (64 or 128 columns) x 4 tiles, level chunks
  const WorkItem *wl_wind;   // wind_cols columns x kWindWarps*wind_rows rows, levels
  const WorkItem *wl_solve;  // row segments of solve_segment columns
  const WorkItem *wl_vert;   // vert_x x vert_y column tiles, R fields
  const WorkItem *wl_vinc;   // the same, the two double-float fields
  const WorkItem *wl_h;      // horizontal WAF tiles (shape waf_tile), levels
  const WorkItem *wl_hinc;   // increment-form WAF tiles, levels
  int n_pt, n_v4, n_vec, n_wind, n_solve, n_vert, n_vinc, n_h, n_hinc;
};

// Tile shapes of the horizontal WAF kernels
inline int waf_tile(const LaunchGeom &L) { return L.htile >= 0 ? L.htile : L.size_tile; }
inline int waf_tile_inc(const LaunchGeom &L) { return L.htile >= 0 ? L.htile : L.size_tile_inc; }

// Launch a kernel of the step (its first statement is grid_begin).  Where a
// step is a few microseconds a kernel (one level a thread, point_levels) the
// launch overlaps the end of the kernel before it: a step of 64x64x30 mixed 127
// us without and 123 with, FP64 247 and 242, of 47x33x23 125 and 119, 193 and
// 189.  From 150x150x40 on nothing changes, and all lose by letting the next
// kernel's blocks in as soon as all blocks of this one have started (64x64x30
// FP64 262 -> 337 us: they settle where there is room, not evenly).
template <class... P, class... A>
void step_launch(const LaunchGeom &L, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                 A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = L.lv == 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Packed FP64 arrays (Fortran extents nj x ni x nk) in the staging buffer and
// the fields in the padded layout that they go to: FP64, FP32, or, with a
// plane size, double-float (high parts, then low parts nplane floats on).
struct UnpackList {
  static constexpr int kMax = 24;
  struct Item {
    const double *src;
    void *dst;
    size_t nplane;
    int nj, ni, nk, f64;
  } it[kMax];
  int n;
};

// Constants of the derived time-invariant fields (bind_cross, bind_wind)
struct BindPar {
  double dtrdz_adv;  // 0.5*dtstepa/dzita
  double dtrdz;      // dtsound/dzita
  double zcs;        // dtrdz*R/cv
  double dtrdx, dxrdt, zfz;  // dtsound/dx, dx/dtsound, g*dtsound
  int rot, nspgx;
};

template <class R> struct Launch {
  // one-off kernel attributes (large dynamic shared memory); call before capture
  static cudaError_t configure_sound();
  static cudaError_t configure_advect();
  // ---- sound (Main/mod_moloch.F90:545-765) ----
  static void sound_prep(const LaunchGeom &L, const Dom<R> *d, int advoff, cudaStream_t s);
  static void sound_div(const LaunchGeom &L, const Dom<R> *d, int uvoff, cudaStream_t s);
  static void sound_solve(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, bool last,
                          cudaStream_t s);
  static void sound_momentum(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff,
                             cudaStream_t s);
  // ---- advection (Main/mod_moloch.F90:767-1042) ----
  static void adv_prep(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s);
  static void adv_vertical(const LaunchGeom &L, const Dom<R> *d, int advoff, cudaStream_t s);
  static void adv_horizontal(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff,
                             cudaStream_t s);
  // theta_v and Exner of a mixed member (double-float, increment form)
  static void adv_vertical_inc(const LaunchGeom &L, const Dom<R> *d, int advoff, cudaStream_t s);
  static void adv_horizontal_inc(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff,
                                 cudaStream_t s);
  static void adv_species_copy(const LaunchGeom &L, const Dom<R> *d, int advoff, cudaStream_t s);
  static void adv_curvature(const LaunchGeom &L, const Dom<R> *d, int advoff, cudaStream_t s);
  static void adv_back(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s);
  // ---- step end (Main/mod_moloch.F90:340-446, mod_bdycod.F90) ----
  static void bdy_ring(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s);
  static void end_relax(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s);
  static void bdy_spectral(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s);
  // a whole step's end without spectral nudging: the pointwise work, then the
  // winds (a mixed member's end in the other half of their pairs)
  static void end_point(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s);
  // ... of the ring and the relaxation zone
  static void end_frame(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s);
  static void end_uvx(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s);
  static void end_winds(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s);
  static void end_cross(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s);
  // the step split at the physics: k_end_ps and the cross-point work up to
  // mkslice (post = false), or status_update with the tendencies (post = true)
  static void end_cross_split(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, bool post,
                              cudaStream_t s);
  static void end_uvstag(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s);
  // status_update of the TKE (ibltyp = 2): tendency (split step) and floor
  static void end_tke(const LaunchGeom &L, const Dom<R> *d, bool whole_step, cudaStream_t s);
  // form_ps: ps from the virtual temperatures end_point left; advance: the
  // last block also advances the clock and the roles (else end_advance does)
  static void end_reduce(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, bool form_ps, bool advance,
                         cudaStream_t s);
  static void end_advance(const LaunchGeom &L, const Dom<R> *d, int uvoff, int advoff, cudaStream_t s);
  // ---- layout conversion (one member, from the host) ----
  // the 3-D fields derived from the bound ones (fmz, fmzf: of row pitch fp and
  // plane fps; the 1-D and 2-D fields and, for FP64, rfmzu and rfmzv in place)
  static void bind_derived(const Stat<R> &sa, const Geom &g, const double *fmz, const double *fmzf,
                           size_t fp, size_t fps, const BindPar &b, cudaStream_t s);
  static void unpack(const UnpackList &l, const Geom &g, cudaStream_t s);
  static void pack3(const R *src, double *dst, const Geom &g, int nj, int ni, int nk,
                    cudaStream_t s);
  // double-float planes (hi, lo) of nplane elements each
  static void pack3_df(const double *src, double *dst, const Geom &g, int nj, int ni, int nk,
                       size_t nplane, cudaStream_t s);
};

// Reduction blocks the mass budget uses for a geometry.
int reduce_blocks(const Geom &g);

}  // namespace mlc
