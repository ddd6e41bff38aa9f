// Binary32 3D 7-point heat half-sweep with plain loads, any alignment; the point
// arithmetic and its order are heat_core.cuh's.
//
// A warp owns 30 columns of 2P rows (lanes 1 .. 30 of 32) and streams along axis 0
// with three planes of them in registers.  Rows r and r + P of a lane are the two
// halves of a packed operation, so that every neighbour of a pair is a pair: axis 0
// and 1 from the lane's own registers (but for the row on either side of its 2P, which
// it loads with its own), axis 2 by shuffle.  No shared memory, no barrier; a plane's
// loads are issued one plane ahead.
//
// Bound by the L2 while both arrays lie in it: a half-sweep of 211 x 173 x 301 takes
// 14.5 us, 88 MB in and out (8 B a point) at 6.1 TB/s.  Staging through shared memory with a barrier
// per plane took 49 us, the TMA ring (rows of 16-byte multiples only) 17.2 at 192^3
// against 10.1 here.  Three pairs a thread (62 registers, 32 warps per SM) measured
// best: at 211 x 173 x 301, TSTEPS=21, 0.704 ms with one, 0.614 two, 0.608 three, 0.638
// four, 0.738 six.
#include <algorithm>
#include <cmath>

#include "heat_core.cuh"
#include "npbgb_common.cuh"

namespace npbgb {

extern int64_t g_cfg_heat_chunk;

namespace {

constexpr int kStrip = 30;  // columns a warp writes
constexpr int kW = 4;       // warps per CTA, one above the other along axis 1
constexpr int P = 3;        // pairs a thread

__device__ __forceinline__ F2 up1(F2 a) {  // from the lane before
  return f2(__shfl_up_sync(0xffffffffu, f2x(a), 1), __shfl_up_sync(0xffffffffu, f2y(a), 1));
}
__device__ __forceinline__ F2 down1(F2 a) {
  return f2(__shfl_down_sync(0xffffffffu, f2x(a), 1), __shfl_down_sync(0xffffffffu, f2y(a), 1));
}

__global__ void __launch_bounds__(32 * kW, 32 / kW)
heat3d_rows(const float* __restrict__ src, float* __restrict__ dst, int64_t n0, int64_t n1, int64_t n2, int chunk) {
  pdl_begin();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t k = int64_t(blockIdx.x) * kStrip + lane;
  const int64_t j0 = 1 + (int64_t(blockIdx.y) * kW + warp) * (2 * P);
  if (j0 >= n1 - 1) return;
  const int64_t ib = 1 + int64_t(blockIdx.z) * chunk;
  const int count = int((ib + chunk < n0 - 1 ? ib + chunk : n0 - 1) - ib);
  const int64_t s0 = n1 * n2;
  const bool out = lane >= 1 && lane <= kStrip && k < n2 - 1;
  // Offsets in a plane of rows j0 - 1 .. j0 + 2P; rows and columns outside the array
  // read its last ones and are not written.
  const int64_t kk = k < n2 ? k : n2 - 1;
  uint32_t off[2 * P + 2];
#pragma unroll
  for (int r = 0; r < 2 * P + 2; ++r) off[r] = uint32_t((j0 - 1 + r < n1 ? j0 - 1 + r : n1 - 1) * n2 + kk);
  const int rows = int(n1 - 1 - j0 < 2 * P ? n1 - 1 - j0 : 2 * P);  // to write

  struct Plane {
    F2 x[P];
    float above, below;
  };
  auto load = [&](const float* p, Plane& v) {
#pragma unroll
    for (int r = 0; r < P; ++r) v.x[r] = f2(p[off[1 + r]], p[off[1 + P + r]]);
    v.above = p[off[0]];
    v.below = p[off[2 * P + 1]];
  };
  const float* p = src + (ib - 1) * s0;
  float* o = dst + ib * s0;
  Plane a, b, c, next;
  load(p, a);
  load(p + s0, b);
  p += 2 * s0;
  load(p, next);
  int left = count;
  // Plane of results from the planes before (im), at (c) and after (ip, the one loaded
  // last); loads the one after that.
  auto step = [&](const Plane& im, const Plane& at, Plane& ip) -> bool {
    ip = next;
    p += s0;
    if (left > 1) load(p, next);
#pragma unroll
    for (int r = 0; r < P; ++r) {
      const F2 jm = r > 0 ? at.x[r > 0 ? r - 1 : 0] : f2(at.above, f2x(at.x[P - 1]));
      const F2 jp = r + 1 < P ? at.x[r + 1 < P ? r + 1 : r] : f2(f2y(at.x[0]), at.below);
      const F2 v = hcore::heat_point2(at.x[r], ip.x[r], im.x[r], jp, jm, down1(at.x[r]), up1(at.x[r]));
      if (out && r < rows) o[off[1 + r]] = f2x(v);
      if (out && r + P < rows) o[off[1 + P + r]] = f2y(v);
    }
    o += s0;
    return --left > 0;
  };
  while (step(a, b, c) && step(b, c, a) && step(c, a, b)) {
  }
}

// Planes per warp: 1.6 sqrt(q), q the planes per warp that the GPU holds at once, at
// most 5, or 4 where the arrays exceed the L2.  Measured best: 1 at q = 0.1 to 1.2
// (45^3, 64^3, 96^3), 2 to 3 at 2 to 4 (128^3, TSTEPS=40: 0.380 ms with 3, 0.426 with
// 4), 5 at 9 to 36 (192^3: 0.607, 10 0.646), 4 at 256^3 (1.139, 5 1.164) and 384^3.
int chunk_of(int64_t n0, int64_t n1, int64_t n2) {
  if (g_cfg_heat_chunk > 0) return int(std::min<int64_t>(g_cfg_heat_chunk, n0 - 2));
  const double q = double(cdiv(n2 - 2, kStrip)) * double(cdiv(n1 - 2, 2 * P)) * double(n0 - 2) / (32.0 * sm_count());
  const int64_t most = n0 * n1 * n2 * 8 > (int64_t(120) << 20) ? 4 : 5;
  const int64_t c = std::max<int64_t>(std::min<int64_t>(int64_t(1.6 * std::sqrt(q) + 0.5), most), 1);
  return int(std::min(std::max(c, cdiv(n0 - 2, 65535)), n0 - 2));
}

}  // namespace

// NPBGB_ERR_STATE (nothing launched) when a plane exceeds the kernel's 32-bit offsets
// or a grid dimension is too large.
int32_t heat3d_rows_run(float* a, float* b, int64_t n0, int64_t n1, int64_t n2, int32_t tsteps, cudaStream_t st) {
  if (n0 > 0x7fffffff || n1 > 0x7fffffff || n2 > 0x7fffffff || n1 * n2 >= (int64_t(1) << 31)) return NPBGB_ERR_STATE;
  const int chunk = chunk_of(n0, n1, n2);
  const int64_t gy = cdiv(n1 - 2, 2 * P * kW), gz = cdiv(n0 - 2, chunk);
  if (gy > 65535 || gz > 65535) return NPBGB_ERR_STATE;
  const dim3 grid{unsigned(cdiv(n2 - 2, kStrip)), unsigned(gy), unsigned(gz)};
  cudaError_t e = cudaSuccess;
  for (int32_t t = 1; t < tsteps && e == cudaSuccess; ++t) {
    e = launch_chained(heat3d_rows, grid, dim3{32u * kW}, 0, st, a, b, n0, n1, n2, chunk);
    if (e == cudaSuccess) e = launch_chained(heat3d_rows, grid, dim3{32u * kW}, 0, st, b, a, n0, n1, n2, chunk);
  }
  return cuda_status(e, "heat3d_rows");
}

}  // namespace npbgb
