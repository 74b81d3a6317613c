// mlc_noalloc.cu -- the mass budget of one domain without any allocation.
//
// Who needs this: a host model that keeps its fields in device memory it
// manages itself (a Fortran/OpenACC model whose memory manager owns the
// device heap, a pool that must not fragment, code that runs where
// cudaMalloc is not allowed, such as inside a callback or a region being
// captured into a graph) can hand the library pointers to its own arrays
// but cannot let the library call cudaMalloc for scratch.  This entry point
// computes the same sums as the budget of mlc_step (Main/mod_massck.F90:
// 77-170) from caller-owned device arrays, keeping its per-block partial
// sums in the file-scope device array below instead of allocating them.
//
// Limits and sharing rules:
// * a domain may have at most kBudgetRows = 32768 rows ((iy-1) * kz); larger
//   domains are rejected with MLC_ERR_TOO_LARGE (what callers rely on to fall
//   back; the array no longer depends on it: one record a block, whatever the
//   rows);
// * every GPU that loads the library holds the 29 KB array until exit;
// * all calls share the one array: calls whose kernels overlap on the GPU
//   (different streams, or different host threads) race on it; serialise
//   them (one stream, or events);
// * every partial record the final pass reads is written by the same call
//   before it is read, so no part of the array has to start at zero.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

#include "../../include/moloch_gb300.h"

namespace {

constexpr long long kBudgetRows = 32768;
constexpr int kBudgetRecord = 8;  // dry, dryadv, qmass, qadv, ps max, ps min, bad, pad
constexpr int kBudgetThreads = 256;
constexpr int kMaxDevices = 64;
// Blocks an SM the rows are dealt to: with 3 every warp of the 512x512x41
// domain takes 6 rows and the blocks are resident at once (178 us; 1: 371,
// 2: 212, 4: 208, 8: 196, the reduction's tail growing with the blocks).
constexpr int kBudgetBlocksSM = 3;
constexpr int kBudgetBlocks = 152 * kBudgetBlocksSM;  // at most

static __device__ __align__(256) double g_budget_scratch[kBudgetBlocks * kBudgetRecord];

// Host-side copy of the array's device address, per device, with the id of
// the CUDA context it was taken in.  In host code the name g_budget_scratch
// is only a stand-in: its device address comes from cudaGetSymbolAddress
// with the device current.  A cudaDeviceReset (or any new primary context)
// reloads the module at another address, so the cached address is used only
// while the current context's id is the one it was taken in; otherwise it is
// looked up again.
std::mutex g_mu;
double *g_scratch_ptr[kMaxDevices] = {};
unsigned long long g_scratch_ctx[kMaxDevices] = {};

// The unique id of the current CUDA context (0 if it cannot be read), from
// driver entry points fetched through the runtime (no link against libcuda).
unsigned long long current_context_id() {
  static PFN_cuCtxGetCurrent_v4000 get_ctx = nullptr;
  static PFN_cuCtxGetId_v12000 get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 4000, cudaEnableDefault, &q) ==
            cudaSuccess && q == cudaDriverEntryPointSuccess)
      get_ctx = reinterpret_cast<PFN_cuCtxGetCurrent_v4000>(p);
    p = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess && q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<PFN_cuCtxGetId_v12000>(p);
    cudaGetLastError();
  });
  if (!get_ctx || !get_id) return 0;
  CUcontext c = nullptr;
  unsigned long long id = 0;
  if (get_ctx(&c) != CUDA_SUCCESS || !c) return 0;
  if (get_id(c, &id) != CUDA_SUCCESS) return 0;
  return id;
}

int scratch_for_current_device(double **out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return MLC_ERR_NODEVICE;
  if (dev < 0 || dev >= kMaxDevices) return MLC_ERR_INVALID;
  const unsigned long long ctx = current_context_id();
  std::lock_guard<std::mutex> lock(g_mu);
  if (!g_scratch_ptr[dev] || ctx == 0 || g_scratch_ctx[dev] != ctx) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_budget_scratch);
    if (e != cudaSuccess || !p) {
      cudaGetLastError();
      return MLC_ERR_CUDA;
    }
    g_scratch_ptr[dev] = static_cast<double *>(p);
    // the lookup makes the device's primary context current if none was
    g_scratch_ctx[dev] = ctx ? ctx : current_context_id();
  }
  *out = g_scratch_ptr[dev];
  return MLC_OK;
}

// The block's sums and extrema, in warp order (a fixed order), by thread 0.
struct Budget {
  double dry, dadv, qm, qadv, pmax, pmin;
  int bad;
};
__device__ __forceinline__ Budget budget_zero() { return {0, 0, 0, 0, -INFINITY, INFINITY, 0}; }
__device__ __forceinline__ void budget_add(Budget &a, const Budget &b) {
  a.dry += b.dry; a.dadv += b.dadv; a.qm += b.qm; a.qadv += b.qadv;
  a.pmax = fmax(a.pmax, b.pmax); a.pmin = fmin(a.pmin, b.pmin);
  a.bad |= b.bad;
}
__device__ Budget block_budget(Budget a) {
  __shared__ Budget sh[kBudgetThreads / 32];
  const unsigned full = 0xffffffffu;
  for (int off = 16; off > 0; off >>= 1) {
    const Budget b{__shfl_down_sync(full, a.dry, off),  __shfl_down_sync(full, a.dadv, off),
                   __shfl_down_sync(full, a.qm, off),   __shfl_down_sync(full, a.qadv, off),
                   __shfl_down_sync(full, a.pmax, off), __shfl_down_sync(full, a.pmin, off),
                   __shfl_down_sync(full, a.bad, off)};
    budget_add(a, b);
  }
  if ((threadIdx.x & 31u) == 0) sh[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < kBudgetThreads / 32; ++w) budget_add(a, sh[w]);
  return a;
}

// Arrays are in the packed reference layout: cross (jx-1, iy-1, kz),
// u (jx, iy-1, kz), v (jx-1, iy, kz), qx (jx-1, iy-1, kz, nqx), ps (jx-1, iy-1).
//
// Pieces of interior rows (i, k) go to warps, `per` in turn each, lanes along j
// (rows start on 8 bytes only, so wider loads are not possible).  A piece is a
// whole row unless there are fewer rows than warps (two rows of 30000 columns
// took 1.6 ms by whole rows).  dx^2 is applied to the sums and the species of a
// point are added before they are weighted by dz*rho: 2 + nqx
// FP64 instructions a point.  On GB300, whose FP64 pipe runs two a clock and
// SM, that pipe bounds the kernel (142 us at 512x512x41 with 5 species; the
// 0.6 GB of loads need 89 us); the form with each species weighted by itself
// needed 23 a point.  The lateral fluxes and the ps extrema are grid-stride
// loops over their own items.  Measured, both kernels, 512x512x41, 5 species:
// 1.71 ms before, 0.18 ms now.
// NQ: species (0: nqx at run time).
template <int NQ>
__global__ void __launch_bounds__(kBudgetThreads) k_budget_partial(
    int jx, int iy, int kz, int nqx, double dx, double dt, int pieces, int per, const double *__restrict__ rho,
    const double *__restrict__ dz, const double *__restrict__ qx, const double *__restrict__ u,
    const double *__restrict__ v, const double *__restrict__ ps, double *scratch) {
  const int nc = jx - 1, nq = NQ > 0 ? NQ : nqx;
  const size_t c2 = (size_t)nc * (iy - 1);
  const size_t c3 = c2 * kz;
  Budget a = budget_zero();
  const int lane = (int)(threadIdx.x & 31u);
  const int warp = (int)(blockIdx.x * (kBudgetThreads / 32) + (threadIdx.x >> 5));
  const int ni = iy - 3, items = ni * kz * pieces;
  const int len = ((nc - 2 + 31) / 32 + pieces - 1) / pieces * 32;  // columns of a piece
  const int t1 = min(items, (warp + 1) * per);
  for (int t = warp * per; t < t1; ++t) {
    const int r = t / pieces, j0 = 1 + (t - r * pieces) * len, j1 = min(nc - 2, j0 + len - 1);
    const int k = r / ni, i = r - k * ni + 1;  // 0-based level and row
    const size_t o0 = c2 * k + (size_t)nc * i;
#pragma unroll 1  // unrolled by 4 (the compiler's choice) 211 us instead of 178
    for (int j = j0 + lane; j <= j1; j += 32) {
      const size_t o = o0 + j;
      const double m = dz[o] * rho[o];
      double q = qx[o];
#pragma unroll
      for (int n = 1; n < nq; ++n) q += qx[o + n * c3];
      a.dry += m;
      a.qm += q * m;
    }
  }
  a.dry *= dx * dx;
  a.qm *= dx * dx;
  const int gt = (int)(blockIdx.x * kBudgetThreads + threadIdx.x), gs = (int)(gridDim.x * kBudgetThreads);
  // flux through one face of the cross point at o: sign * wind * dt*dx*dz*rho
  auto face = [&](size_t o, double wind) {
    const double f = wind * dt * dx * dz[o] * rho[o];
    double q = qx[o];
    for (int n = 1; n < nq; ++n) q += qx[o + n * c3];
    a.dadv += f;
    a.qadv += q * f;
  };
  // west (u at 1, in) and east (u at jx, out) columns of every row
  for (int e = gt; e < (iy - 1) * kz; e += gs) {
    face((size_t)nc * e, u[(size_t)jx * e]);
    face((size_t)nc * e + nc - 1, -u[(size_t)jx * e + jx - 1]);
  }
  // the south and north rows and ps by warps, 32 columns of a row at a time
  const int chunks = (jx - 3 + 31) / 32, nwarp = (int)(gridDim.x * (kBudgetThreads / 32));
  // south (v at 1, in) and north (v at iy, out) rows, j in jci
  for (int e = warp; e < chunks * kz; e += nwarp) {
    const int k = e / chunks, j = (e - k * chunks) * 32 + lane + 1;
    if (j > nc - 2) continue;
    const size_t ov = (size_t)nc * iy * k + j;
    face(c2 * k + j, v[ov]);
    face(c2 * k + (size_t)nc * (iy - 2) + j, -v[ov + (size_t)nc * (iy - 1)]);
  }
  for (int e = warp; e < chunks * ni; e += nwarp) {
    const int i = e / chunks, j = (e - i * chunks) * 32 + lane + 1;
    if (j > nc - 2) continue;
    const double x = ps[(size_t)nc * (i + 1) + j];
    if (!isfinite(x)) a.bad = 1;
    else { a.pmax = fmax(a.pmax, x); a.pmin = fmin(a.pmin, x); }
  }
  a = block_budget(a);
  if (threadIdx.x == 0) {
    double *rec = scratch + (size_t)blockIdx.x * kBudgetRecord;
    rec[0] = a.dry; rec[1] = a.dadv; rec[2] = a.qm; rec[3] = a.qadv;
    rec[4] = a.pmax; rec[5] = a.pmin; rec[6] = a.bad; rec[7] = 0.0;
  }
}

// One block adds the records, a few a thread in record order, then as the
// blocks do (one thread adding them all took 1.4 ms of a 1.7 ms call).
__global__ void __launch_bounds__(kBudgetThreads) k_budget_final(const double *scratch, int nblocks, double *out) {
  Budget a = budget_zero();
  for (int b = (int)threadIdx.x; b < nblocks; b += kBudgetThreads) {
    const double *rec = scratch + (size_t)b * kBudgetRecord;
    budget_add(a, Budget{rec[0], rec[1], rec[2], rec[3], rec[4], rec[5], rec[6] != 0.0});
  }
  a = block_budget(a);
  if (threadIdx.x != 0) return;
  out[0] = a.dry; out[1] = a.dadv; out[2] = a.qm; out[3] = a.qadv;
  out[4] = a.bad ? NAN : a.pmax;
  out[5] = a.bad ? NAN : a.pmin;
  out[6] = a.bad ? 1.0 : 0.0;
}

}  // namespace

extern "C" int mlc_mass_budget_noalloc(const mlc_dims *d, double dx, double dt,
                                       const double *rho, const double *dz, const double *qx,
                                       const double *u, const double *v, const double *ps,
                                       double *out, void *stream) {
  if (!d || !rho || !dz || !qx || !u || !v || !ps || !out) return MLC_ERR_INVALID;
  if (d->jx < 5 || d->iy < 5 || d->kz < 1 || d->nqx < 1) return MLC_ERR_INVALID;
  const long long nrows = (long long)(d->iy - 1) * d->kz;
  if (nrows > kBudgetRows) return MLC_ERR_TOO_LARGE;
  double *scratch = nullptr;
  const int st = scratch_for_current_device(&scratch);
  if (st != MLC_OK) return st;
  // pieces a warp: as few as fill kBudgetBlocksSM blocks on each of 152 SMs
  constexpr int kWarps = kBudgetThreads / 32, kFull = kBudgetBlocks * kWarps;
  const int rows = (d->iy - 3) * d->kz, chunks = (d->jx - 3 + 31) / 32;
  const int pieces = rows >= kFull ? 1 : std::min(chunks, kFull / rows);
  const int items = rows * pieces, per = (items + kFull - 1) / kFull;
  const int nblocks = (items + per * kWarps - 1) / (per * kWarps);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  auto part = d->nqx == 5 ? k_budget_partial<5> : d->nqx == 2 ? k_budget_partial<2> : k_budget_partial<0>;
  part<<<nblocks, kBudgetThreads, 0, s>>>(d->jx, d->iy, d->kz, d->nqx, dx, dt, pieces, per, rho, dz, qx, u, v, ps,
                                       scratch);
  k_budget_final<<<1, kBudgetThreads, 0, s>>>(scratch, nblocks, out);
  return cudaGetLastError() == cudaSuccess ? MLC_OK : MLC_ERR_CUDA;
}
