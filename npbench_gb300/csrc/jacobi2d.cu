// 2D 5-point Jacobi time loop (polybench/jacobi_2d/jacobi_2d_numpy.py:4-10).
//
// Per interior point, in the reference's order:
//   dst = 0.2 * ((((c + w) + e) + s) + n)
// with w/e the column neighbours j-1/j+1 and s/n the row neighbours i+1/i-1.
//
// Kernel layout (one launch per half-sweep): every warp owns a strip of 32
// columns and streams down a chunk of rows (jacobi_core.cuh: rows i-1, i,
// i+1 in registers, w/e neighbours by shuffle, kUnroll rows loaded ahead).
// Warps never wait on each other.
//
// binary32 uses IEEE float operations.  binary64 runs in binary32 limbs
// (jacobi_limb.cuh) or, where a setting asks for it, its four additions
// exactly in fixed point on the integer pipe (fx64.cuh) for every point whose
// five inputs lie in [2^-7, 1) or are +0 (refused values carry a poison bit),
// and uses hardware binary64 for any other point.  The fixed-point points also
// take the final product by 0.2 on the integer pipes (fx::mul02: the exact
// integer product of the significands, rounded once to nearest even), so they
// leave the binary64 pipe to the hardware warps.  Both paths give the IEEE
// result bit for bit.
#include <algorithm>
#include <cmath>

#include "jacobi_core.cuh"
#include "jacobi_limb.cuh"
#include "tma.cuh"

namespace npbgb {

extern int64_t g_cfg_f64_emulation;
extern int64_t g_cfg_jacobi_chunk;
extern int64_t g_cfg_jacobi_hw_warps;
extern int64_t g_cfg_jacobi_fx_mul;
extern int64_t g_cfg_jacobi_fx_adds;
extern int64_t g_cfg_jacobi_tma;
extern int64_t g_cfg_jacobi_bands;

cudaError_t scratch_pool(cudaMemPool_t* out);  // jacobi_bands.cu

template <typename T>
int32_t jacobi2d_bands_run(T* a, T* b, int64_t ny, int64_t nx, int32_t tsteps, cudaStream_t st);

namespace {

constexpr int kWarps = 8;
constexpr int kUnroll = 4;

// Grid: x over groups of kWarps column strips, y over chunks of rows.  With
// FX, warps below hw_warps take the hardware binary64 path so that the
// binary64 pipe works next to the integer pipe (same results either way).
template <typename T, bool FX, int MAD, bool IMUL, bool HWIMUL>
__global__ void __launch_bounds__(32 * kWarps)
jacobi2d_strip(const T* __restrict__ src, T* __restrict__ dst, int64_t ny, int64_t nx, int chunk,
               int hw_warps, uint32_t one) {
  pdl_begin();
  const int warp = threadIdx.x >> 5;
  const int64_t k0 = 1 + (int64_t(blockIdx.x) * kWarps + warp) * 32;
  if (k0 >= nx - 1) return;  // whole strip outside the interior (warp-uniform)
  const int64_t ib = 1 + int64_t(blockIdx.y) * chunk;
  const int64_t ie = (ib + chunk < ny - 1) ? ib + chunk : ny - 1;
  // Rows loaded ahead: 4 for binary32; 1 for binary64, whose chunks are short
  // (2 ahead measured 5-10% slower at 500^2 to 4096^2 with 4 hardware warps).
  if (FX && warp < hw_warps)
    jcore::strip_rows<T, false, false, 1, 0, true, HWIMUL>(src, dst, nx, k0, ib, ie, one);
  else
    jcore::strip_rows<T, FX, false, FX ? 1 : kUnroll, MAD, IMUL>(src, dst, nx, k0, ib, ie, one);
}

__device__ unsigned int g_jacobi_tma_error;  // a wait gave up; bit 0: on an mbarrier, 1: on a neighbouring CTA

using jcore::kTmaRing;
using jcore::kTmaRows;
using jcore::tma_strip_rows;
template <typename T>
using TmaStrip = jcore::TmaStrip<T, kWarps>;

template <typename T, bool FX, int MAD, bool IMUL>
__global__ void __launch_bounds__(32 * kWarps)
jacobi2d_tma(const __grid_constant__ CUtensorMap map, const T* __restrict__ src, T* __restrict__ dst,
             int64_t ny, int64_t nx, int chunk, int hw_warps, uint32_t one) {
  pdl_begin();
  using G = TmaStrip<T>;
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5;
  unsigned char* ring = smem + warp * G::kWarpBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kWarps * G::kWarpBytes) + warp * kTmaRing;
  const int64_t k0 = 1 + (int64_t(blockIdx.x) * kWarps + warp) * 32;
  if (k0 >= nx - 1) return;  // whole strip outside the interior (warp-uniform)
  const int64_t ib = 1 + int64_t(blockIdx.y) * chunk;
  const int64_t ie = (ib + chunk < ny - 1) ? ib + chunk : ny - 1;
  if ((threadIdx.x & 31) == 0) {
    for (int b = 0; b < kTmaRing; ++b) tma::mbar_init(&bars[b], 1);
    tma::fence_mbar_init();
  }
  __syncwarp();
  const bool ok = (FX && warp < hw_warps)
                      ? tma_strip_rows<T, false, MAD, IMUL>(&map, src, dst, nx, k0, ib, ie, ring, bars, one)
                      : tma_strip_rows<T, FX, MAD, IMUL>(&map, src, dst, nx, k0, ib, ie, ring, bars, one);
  if (!ok && (threadIdx.x & 31) == 0) atomicOr(&g_jacobi_tma_error, 1u);
}

template <int W>
__device__ __forceinline__ void limb_unit(const double* __restrict__ src, double* __restrict__ dst, int64_t ny,
                                          int64_t nx, int chunk) {
  pdl_begin();
  const int warp = threadIdx.x >> 5;
  const int64_t k0 = 1 + (int64_t(blockIdx.x) * W + warp) * jlimb::kStrip;
  if (k0 >= nx - 1) return;
  const int64_t ib = 1 + int64_t(blockIdx.y) * chunk;
  const int64_t ie = (ib + chunk < ny - 1) ? ib + chunk : ny - 1;
  if (!jlimb::rows(jlimb::Limbs{fxl::consts()}, src, dst, nx, k0, ib, ie))
    jlimb::rows_hardware(src, dst, nx, k0, ib, ie);
}
constexpr int kLimbWarps = 4;
constexpr int kLoopWarps = 25;
constexpr uint64_t kLoopLimitNs = 2000000000ull;
// No least number of CTAs per SM here: any asked for schedules worse (5 to 8%).
__global__ void __launch_bounds__(32 * kLimbWarps)
jacobi2d_limb(const double* __restrict__ src, double* __restrict__ dst, int64_t ny, int64_t nx, int chunk) {
  limb_unit<kLimbWarps>(src, dst, ny, nx, chunk);
}
__global__ void __launch_bounds__(32, 28)
jacobi2d_limb_alone(const double* __restrict__ src, double* __restrict__ dst, int64_t ny, int64_t nx, int chunk) {
  limb_unit<1>(src, dst, ny, nx, chunk);
}

// The whole time loop in one cooperative launch, for small grids: a warp keeps one unit (a
// strip by `chunk` rows, numbered along the rows of strips).  Half-sweep s starts when
// the CTAs with a unit next to one of this CTA's, at most `near` away, have done s of
// them: they then have written what it reads and read what it writes.  Bound by that
// hand-off, about 1.5 us of 3.6 a half-sweep at 400^2 (a release store to the counter
// instead of the reduction: 4.5).
__global__ void __launch_bounds__(32 * kLoopWarps, 1)
jacobi2d_limb_loop(double* a, double* b, int64_t ny, int64_t nx, int halfsweeps, int strips,
                   int chunk, int units, int near, uint32_t* __restrict__ done) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit = int(blockIdx.x) * int(blockDim.x >> 5) + warp;
  const int64_t k0 = 1 + int64_t(unit % strips) * jlimb::kStrip, ib = 1 + int64_t(unit / strips) * chunk;
  const int64_t ie = ib + chunk < ny - 1 ? ib + chunk : ny - 1;
  const int cta = int(blockIdx.x) - near + lane;
  const bool waits = warp == 0 && lane <= 2 * near && lane != near && cta >= 0 && cta < int(gridDim.x);
  const jlimb::Limbs limbs{fxl::consts()};
  for (int s = 0; s < halfsweeps; ++s) {
    bool ok = true;
    if (s > 0 && waits) {
      uint64_t t0 = 0;
      for (uint32_t n = 1;; ++n) {
        uint32_t v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(done + cta) : "memory");
        if (int32_t(v - uint32_t(s)) >= 0) break;
        if ((n & 255u) == 0) {
          const uint64_t now = tma::globaltimer();
          if (t0 == 0) t0 = now;
          if (now - t0 > kLoopLimitNs) {
            atomicOr(&g_jacobi_tma_error, 2u);
            ok = false;
            break;
          }
        }
      }
    }
    if (__syncthreads_or(!ok)) return;
    const double* src = s & 1 ? b : a;
    double* dst = s & 1 ? a : b;
    if (unit < units && !jlimb::rows<jlimb::Limbs, true>(limbs, src, dst, nx, k0, ib, ie))
      jlimb::rows_hardware<true>(src, dst, nx, k0, ib, ie);
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(done + blockIdx.x) : "memory");
  }
}

// Warps per CTA and rows per warp, by q, the strips' rows per warp that the GPU holds at
// once (36 per SM).  From q = 9 a warp is a CTA of its own, with 64 registers instead of
// 56 and no neighbours to wait for at a CTA's end (1700 x 1500, TSTEPS=21: 0.530 ms
// against 0.572; 4096^2, 5: 0.557 / 0.60; but 1000^2, 50: 0.744 / 0.711).  Rows are an
// even number (two at a time) growing with the square root of q.  Measured best with
// four warps at q = 0.1 to 3.06: 2 (600^2, TSTEPS=50: 0.424 ms, 4 0.537; 650^2 0.482 and
// 0.530; 700^2 0.512 and 0.538); 3.1: 4 (1000 x 500: 0.525, 2 0.544); 3.3: 4 (1403 x
// 377: 0.539, 2 0.573, 6 0.652); 6.2: 6 (1000^2: 0.715, 4 0.739, 8 0.795); with one at
// 15: 10 to 16; 30: 16 to 24; 48: 20 (2800^2, 11: 0.707, 10 0.736); 102: 24 to 32.
struct LimbShape { int warps, chunk; };
LimbShape limb_shape(int64_t ny, int64_t nx) {
  const double q = double(cdiv(nx - 2, jlimb::kStrip)) * double(ny - 2) / (36.0 * sm_count());
  const bool alone = q >= 9.0;
  const int64_t least = cdiv(ny - 2, 65535);  // the grid's limit
  if (g_cfg_jacobi_chunk > 0) return {alone ? 1 : kLimbWarps, int(std::max<int64_t>(g_cfg_jacobi_chunk, least))};
  const int64_t pairs = alone ? int64_t(1.5 * std::sqrt(q) + 0.5) : q < 3.08 ? 1 : int64_t(1.2 * std::sqrt(q) + 0.15);
  return {alone ? 1 : kLimbWarps, int(std::max<int64_t>(2 * pairs, least + (least & 1)))};
}

// Binary64 in limbs (jacobi_limb.cuh).  Bound by instructions on large grids, by a
// launch's latency on small ones.  Against the fixed-point strips and the TMA ring
// with their best settings (ms, TSTEPS=50, 11 at 2800^2 and 4096^2; then NPBench's
// initial field, whose values leave [0, 1)): 300^2 0.356 to 0.29 and 0.49 to 0.34;
// 1000^2 0.84 to 0.715 and 1.31 to 0.74; 2800^2 0.95 to 0.71 and 1.80 to 0.72; 4096^2
// 1.71 to 1.39 and 3.41 to 1.40.
int32_t run_limb(double* a, double* b, int64_t ny, int64_t nx, int32_t tsteps, cudaStream_t st) {
  const LimbShape s = limb_shape(ny, nx);
  const auto kern = s.warps == 1 ? jacobi2d_limb_alone : jacobi2d_limb;
  const dim3 grid{unsigned(cdiv(nx - 2, s.warps * jlimb::kStrip)), unsigned(cdiv(ny - 2, s.chunk))};
  cudaError_t e = cudaSuccess;
  for (int32_t t = 1; t < tsteps && e == cudaSuccess; ++t) {
    e = launch_chained(kern, grid, dim3{32u * unsigned(s.warps)}, 0, st, static_cast<const double*>(a), b, ny, nx, s.chunk);
    if (e == cudaSuccess)
      e = launch_chained(kern, grid, dim3{32u * unsigned(s.warps)}, 0, st, static_cast<const double*>(b), a, ny, nx, s.chunk);
  }
  return cuda_status(e, "jacobi2d_limb");
}

// NPBGB_ERR_STATE (nothing launched) where the chained launches are to be used.  The line
// follows the units a CTA; in us, chained and in one launch, values in [0, 1) and then
// standard normal ones: 2 (150^2, TSTEPS=50) 244, 274 and 306, 345; 10 (200 x 481, 20)
// 147, 138 and 191, 166; 14 (350^2, 50) 377, 329 and 514, 413; 16 (300 x 481, 50) 342, 328
// and 485, 437; 18 (400^2, 50) 391, 349 and 518, 466; 25 (480^2, 50) 412, 409 and 541, 548;
// 32 (608 x 481, 30) 244, 274 and 325, 379.  Wider grids do not gain: 150 x 1000, 30, 197,
// 229 and 269, 286; 200 x 700 212, 213 and 294, 277.
int32_t run_limb_loop(double* a, double* b, int64_t ny, int64_t nx, int32_t tsteps, cudaStream_t st) {
  if (g_cfg_jacobi_bands != 1 || g_cfg_jacobi_chunk != 0 || tsteps < 16 || tsteps > (1 << 30) || queue_exists())
    return NPBGB_ERR_STATE;
  constexpr int kChunk = 2;
  const int64_t strips = cdiv(nx - 2, jlimb::kStrip), units = strips * cdiv(ny - 2, kChunk);
  if (nx > 481 || units < 10 * int64_t(sm_count()) || units > kLoopWarps * int64_t(sm_count())) return NPBGB_ERR_STATE;
  const int per_cta = int(cdiv(units, sm_count()));
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone)
    return NPBGB_ERR_STATE;  // (the chained launches need no scratch memory)
  const int nb = int(cdiv(units, per_cta)), near = int(cdiv(strips + 1, per_cta));
  cudaMemPool_t pool;
  void* scratch = nullptr;
  cudaError_t e;
  if ((e = scratch_pool(&pool)) != cudaSuccess ||
      (e = cudaMallocFromPoolAsync(&scratch, size_t(nb) * sizeof(uint32_t), pool, st)) != cudaSuccess) {
    cudaGetLastError();
    return NPBGB_ERR_STATE;
  }
  e = cudaMemsetAsync(scratch, 0, size_t(nb) * sizeof(uint32_t), st);
  if (e == cudaSuccess) {
    auto* done = static_cast<uint32_t*>(scratch);
    int hs = 2 * (tsteps - 1), strips_ = int(strips), chunk = kChunk, units_ = int(units), near_ = near;
    void* args[] = {&a, &b, &ny, &nx, &hs, &strips_, &chunk, &units_, &near_, &done};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(nb));
    cfg.blockDim = dim3(32u * unsigned(per_cta));
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = launch_together(cfg, reinterpret_cast<const void*>(jacobi2d_limb_loop), args);
  }
  cudaFreeAsync(scratch, st);
  return e == cudaSuccess ? NPBGB_OK : NPBGB_ERR_STATE;  // not launched
}

int pick_chunk(int64_t ny, int64_t col_blocks) {
  if (g_cfg_jacobi_chunk > 0) return int(g_cfg_jacobi_chunk);
  // About 16 warps per SM over 152 SMs, rows per warp at least 3 (small
  // grids want short chunks for enough CTAs: 3-4 rows measured best at 500^2
  // and 1000^2, the computed chunk at 2000^2 and 4096^2).
  const int64_t target_blocks = int64_t(sm_count()) * 16 / kWarps * 4;
  int64_t chunks = cdiv(target_blocks, col_blocks > 0 ? col_blocks : 1);
  int64_t c = cdiv(ny - 2, chunks > 0 ? chunks : 1);
  if (c < 3) c = 3;
  if (c > ny - 2) c = ny - 2;
  return int(c);
}

// The chained half-sweeps with the TMA kernel; NPBGB_ERR_STATE (nothing
// launched) when the arrays do not meet TMA's rules (16-byte aligned base and
// rows) or a form other than plain integer additions is asked for.
template <typename T, bool FX>
int32_t run_tma(T* a, T* b, int64_t ny, int64_t nx, int32_t tsteps, dim3 grid, int chunk, int hw,
                int mad, int64_t im, cudaStream_t st) {
  using G = TmaStrip<T>;
  if (mad != 0 || im == 2) return NPBGB_ERR_STATE;
  if ((nx * int64_t(sizeof(T))) % 16 != 0 || ny > 0x7fffffff || nx > 0x7fffffff) return NPBGB_ERR_STATE;
  CUtensorMap map_a, map_b;
  const uint64_t dims[3] = {uint64_t(nx), uint64_t(ny), 1u};
  const uint32_t box[3] = {uint32_t(G::BX), uint32_t(kTmaRows), 1u};
  if (tma::encode_3d(&map_a, sizeof(T), a, dims, box) != cudaSuccess ||
      tma::encode_3d(&map_b, sizeof(T), b, dims, box) != cudaSuccess)
    return NPBGB_ERR_STATE;
  auto kern = im == 0 ? jacobi2d_tma<T, FX, 0, false> : jacobi2d_tma<T, FX, 0, true>;
  const dim3 block{32u * kWarps};
  cudaError_t e = cudaSuccess;
  for (int32_t t = 1; t < tsteps && e == cudaSuccess; ++t) {
    e = launch_chained(kern, grid, block, G::smem(), st, map_a, a, b, ny, nx, chunk, hw, 1u);
    if (e == cudaSuccess)
      e = launch_chained(kern, grid, block, G::smem(), st, map_b, b, a, ny, nx, chunk, hw, 1u);
  }
  return cuda_status(e, "jacobi2d_tma");
}

template <typename T, bool FX>
int32_t run(T* a, T* b, int64_t ny, int64_t nx, int32_t tsteps, cudaStream_t st) {
  if (tsteps <= 1 || ny < 3 || nx < 3) return NPBGB_OK;
  {
    const int32_t r = jacobi2d_bands_run<T>(a, b, ny, nx, tsteps, st);
    if (r != NPBGB_ERR_STATE) return r;
  }
  if constexpr (FX) {
    // Limbs unless a setting of the other forms asks for one of those.
    if (g_cfg_jacobi_hw_warps < 0 && g_cfg_jacobi_tma != 2 && g_cfg_jacobi_fx_adds == 0 &&
        g_cfg_jacobi_fx_mul == 1) {
      const int32_t r = run_limb_loop(a, b, ny, nx, tsteps, st);
      return r != NPBGB_ERR_STATE ? r : run_limb(a, b, ny, nx, tsteps, st);
    }
  }
  const int64_t gx = cdiv(nx - 2, 32 * kWarps);
  const int chunk = pick_chunk(ny, gx);
  const int64_t gy = cdiv(ny - 2, chunk);
  if (gx > 0x7fffffff || gy > 65535) return set_error(NPBGB_ERR_ARG, "jacobi2d: extent too large");
  const dim3 grid{unsigned(gx), unsigned(gy)};
  const int hw = jacobi_hw_warps();
  const dim3 block{32u * kWarps};
  // Fixed-point additions as plain integer adds (with the integer product by
  // 0.2 they measured fastest at every size: 1000^2 TSTEPS=100 1.83 ms against
  // 1.94 with multiply-add adds and 2.10 with the rounding on the multiply-add
  // pipe) unless NPBGB_CFG_JACOBI_FX_ADDS says otherwise; the product by 0.2 on
  // the integer pipes unless NPBGB_CFG_JACOBI_FX_MUL = 0.
  const int mad = (FX && g_cfg_jacobi_fx_adds > 0) ? int(g_cfg_jacobi_fx_adds) - 1 : 0;
  const int64_t im = g_cfg_jacobi_fx_mul;
  // The TMA ring where it pays: binary64 arrays of 48 MiB and more (the pair
  // beyond most of the L2), automatically; any aligned grid when forced
  // (NPBGB_CFG_JACOBI_TMA = 2).  Measured on GB300 (TSTEPS=21 at 4096^2 and
  // 2800^2, 41 at 2048^2, 100 at 1000^2 and 500^2; best settings of each
  // form, ms): 4096^2 binary64 3.44 against 4.04 with plain loads, 2800^2
  // 1.88 / 1.99; grids the L2 holds lose (2048^2, 32 MiB arrays: 2.11 / 1.92,
  // 1000^2 1.91 / 1.64, 500^2 1.45 / 0.89), and binary32 loses at every size
  // (4096^2 1.68 / 1.16): its plain strips already load four rows ahead.
  const bool big = nx * ny * int64_t(sizeof(T)) >= (int64_t(48) << 20);
  if (g_cfg_jacobi_tma == 2 || (g_cfg_jacobi_tma == 1 && FX && big)) {
    // 16-row chunks and 3 of 8 warps on hardware binary64 measured best with the
    // ring at 4096^2 (3.44 ms; the plain form's 54-row chunks 3.63, 4 warps 3.61).
    const int tchunk = g_cfg_jacobi_chunk > 0 ? int(g_cfg_jacobi_chunk) : (ny - 2 < 16 ? int(ny - 2) : 16);
    const int thw = g_cfg_jacobi_hw_warps >= 0 ? int(g_cfg_jacobi_hw_warps) : 3;
    const int64_t tgy = cdiv(ny - 2, tchunk);
    if (tgy <= 65535) {
      const int32_t r = run_tma<T, FX>(a, b, ny, nx, tsteps, dim3{unsigned(gx), unsigned(tgy)}, tchunk,
                                       thw, mad, im, st);
      if (r != NPBGB_ERR_STATE) return r;
    }
  }
  using Kern = void (*)(const T*, T*, int64_t, int64_t, int, int, uint32_t);
  Kern kern;
  if (mad == 2)
    kern = im == 0 ? jacobi2d_strip<T, FX, 2, false, false>
         : im == 1 ? jacobi2d_strip<T, FX, 2, true, false> : jacobi2d_strip<T, FX, 2, true, true>;
  else if (mad == 1)
    kern = im == 0 ? jacobi2d_strip<T, FX, 1, false, false>
         : im == 1 ? jacobi2d_strip<T, FX, 1, true, false> : jacobi2d_strip<T, FX, 1, true, true>;
  else
    kern = im == 0 ? jacobi2d_strip<T, FX, 0, false, false>
         : im == 1 ? jacobi2d_strip<T, FX, 0, true, false> : jacobi2d_strip<T, FX, 0, true, true>;
  cudaError_t e = cudaSuccess;
  for (int32_t t = 1; t < tsteps && e == cudaSuccess; ++t) {
    e = launch_chained(kern, grid, block, 0, st, a, b, ny, nx, chunk, hw, 1u);
    if (e == cudaSuccess) e = launch_chained(kern, grid, block, 0, st, b, a, ny, nx, chunk, hw, 1u);
  }
  return cuda_status(e, "jacobi2d_strip");
}

}  // namespace

// Reads and clears the TMA kernel's device error word (host; synchronises).
uint32_t take_jacobi_tma_device_error() {
  unsigned int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_jacobi_tma_error, sizeof(v)) != cudaSuccess) return 0xffffffffu;
  if (v) cudaMemcpyToSymbol(g_jacobi_tma_error, &zero, sizeof(zero));
  return v;
}

}  // namespace npbgb

extern "C" int32_t npbgb_jacobi2d(void* A, void* B, int64_t ny, int64_t nx, int32_t tsteps,
                                  int32_t dtype, void* stream) {
  using namespace npbgb;
  if (ny < 0 || nx < 0) return set_error(NPBGB_ERR_ARG, "jacobi2d: negative extent");
  if (tsteps > 1 && ny >= 3 && nx >= 3) {
    if (!A || !B) return set_error(NPBGB_ERR_ARG, "jacobi2d: null array");
    if (A == B) return set_error(NPBGB_ERR_ARG, "jacobi2d: A and B alias");
  }
  cudaStream_t st = as_stream(stream);
  if (dtype == NPBGB_F64) {
    double* a = static_cast<double*>(A);
    double* b = static_cast<double*>(B);
    return g_cfg_f64_emulation ? run<double, true>(a, b, ny, nx, tsteps, st)
                               : run<double, false>(a, b, ny, nx, tsteps, st);
  }
  if (dtype == NPBGB_F32)
    return run<float, false>(static_cast<float*>(A), static_cast<float*>(B), ny, nx, tsteps, st);
  return set_error(NPBGB_ERR_DTYPE, "jacobi2d: dtype %d", dtype);
}
