// Binary32 Jacobi-1D with the whole time loop in one cooperative launch; the point
// arithmetic and its order are jacobi1d.cu's (polybench/jacobi_1d/jacobi_1d_numpy.py:4-8).
//
// A CTA owns w points and computes kSpan >= w + 2H of them redundantly for H
// half-sweeps at a time (the valid part shrinks by a point per side and half-sweep),
// then takes the H points on either side from its neighbours: tagged 8-byte elements
// through L2, so that a launch per H half-sweeps and its ramp-up go away.  Within the
// CTA a warp owns 56 points, two adjacent ones a lane, and computes the four on either
// side redundantly for four half-sweeps at a time; values stay in registers, neighbours
// come by shuffle, and one CTA barrier per four half-sweeps passes the outer points on.
//
// Bound by the latency of a half-sweep's shuffles and its chain of three operations,
// 210 clocks with the exchanges; N=32000, TSTEPS=4000 takes 0.87 ms where a chained
// launch per 48 half-sweeps took 1.34 (a barrier per half-sweep, 3 points a lane), N=3200,
// TSTEPS=800 0.21 / 0.29.  Not for binary64: its three operations a point hold the
// binary64 pipe for 60 clocks per 32 points, so the redundant points cost more than the
// launches saved (4.7 ms against 3.1), and on the integer pipes (fx64.cuh) the chain of a
// point is as long as the whole half-sweep there (3.5 ms).
//
// Every wait is bounded: a neighbour that sends nothing for two seconds sets an error
// word and the kernel ends.
#include <algorithm>

#include "npbgb_common.cuh"
#include "tma.cuh"

namespace npbgb {

cudaError_t scratch_pool(cudaMemPool_t* out);  // jacobi_bands.cu

namespace {

constexpr uint64_t kLimitNs = 2000000000ull;
constexpr int kWarps = 8;
constexpr int kOwn = 56;                  // points of a warp: lanes 2 .. 29
constexpr int kSpan = kWarps * kOwn + 8;  // points of a CTA
constexpr int kInner = 4;                 // half-sweeps between exchanges within the CTA

__device__ unsigned int g_j1_error;  // bit 0: a neighbour wait gave up

using Mail = unsigned long long;  // {tag, value}

__device__ __forceinline__ float point(float w, float c, float e) {
  return mul_rn(0.33333f, add_rn(add_rn(w, c), e));
}

__global__ void __launch_bounds__(32 * kWarps, 1)
jacobi1d_resident(float* __restrict__ A, float* __restrict__ B, int64_t n, int halfsweeps, int w, int H,
                  Mail* __restrict__ mail) {
  constexpr uint32_t kAll = 0xffffffffu;
  __shared__ float edge[2][kWarps][2][4];  // [parity][warp][west, east]: four owned points
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = blockIdx.x, nb = gridDim.x;
  const int64_t first = 1 + int64_t(b) * w - H;  // global index of local point 0
  // Boxes: [CTA][to the west, to the east][parity][H]
  auto box = [&](int cta, int side, int round) { return mail + ((int64_t(cta) * 2 + side) * 2 + (round & 1)) * H; };
  int q[2];
  int64_t g[2];
  bool keep[2], mine[2];     // never changes; written by this lane
  float even[2], odd[2];     // a kept point's values in even and odd fields
  float x[2], before[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    q[i] = warp * kOwn + lane * 2 + i;
    g[i] = first + q[i];
    keep[i] = g[i] < 1 || g[i] >= n - 1;
    const bool owned = q[i] >= H && q[i] < H + w && !keep[i];
    mine[i] = owned && lane >= 2 && lane < 30;
    even[i] = odd[i] = 0.0f;
    if (g[i] == 0 || g[i] == n - 1) even[i] = A[g[i]], odd[i] = B[g[i]];
    x[i] = owned ? A[g[i]] : even[i];
    before[i] = x[i];
  }
  const bool kept = __any_sync(kAll, keep[0] || keep[1]);

  // Rounds of H half-sweeps.  A CTA posts round r + 2 over r after it has taken r + 1
  // from the same neighbour, which sent that after it had taken r.
  int parity = 0, round = 0;
  for (int done = 0; done < halfsweeps; ++round) {
    const uint32_t tag = uint32_t(round) + 1;
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const Mail m = static_cast<Mail>(tag) << 32 | __float_as_uint(x[i]);
      Mail* to[2] = {mine[i] && b > 0 && q[i] < 2 * H ? box(b, 0, round) + (q[i] - H) : nullptr,
                     mine[i] && b < nb - 1 && q[i] >= w ? box(b, 1, round) + (q[i] - w) : nullptr};
#pragma unroll
      for (int side = 0; side < 2; ++side)
        if (to[side]) asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(to[side]), "l"(m) : "memory");
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      // Points past the halo's end only keep its neighbours from odd values.
      const Mail* from = nullptr;
      if (!keep[i] && q[i] < H) from = box(b - 1, 1, round) + q[i];
      if (!keep[i] && q[i] >= H + w) from = box(b + 1, 0, round) + (q[i] - H - w < H ? q[i] - H - w : H - 1);
      if (from) {
        Mail m;
        uint64_t t0 = 0;
        for (uint32_t tries = 1; ok; ++tries) {
          asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(m) : "l"(from) : "memory");
          if (uint32_t(m >> 32) == tag) {
            x[i] = __uint_as_float(uint32_t(m));
            break;
          }
          if ((tries & 255u) == 0) {
            const uint64_t now = tma::globaltimer();
            if (t0 == 0) t0 = now;
            if (now - t0 > kLimitNs) {
              atomicOr(&g_j1_error, 1u);
              ok = false;
            }
          }
        }
      }
    }
    if (__syncthreads_or(!ok)) return;
    const int steps = halfsweeps - done < H ? halfsweeps - done : H;
    for (int s = 0; s < steps; s += kInner) {
      const int k = steps - s < kInner ? steps - s : kInner;  // even, as done and s are
#pragma unroll
      for (int r = 0; r < kInner; ++r) {
        if (r >= k) break;
        const float west = __shfl_up_sync(kAll, x[1], 1), east = __shfl_down_sync(kAll, x[0], 1);
        before[0] = x[0], before[1] = x[1];
        x[0] = point(west, before[0], before[1]);
        x[1] = point(before[0], before[1], east);
        if (kept) {
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (keep[i]) x[i] = (r & 1) == 0 ? odd[i] : even[i];
        }
      }
      if (done + s + k == halfsweeps) break;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (lane == 2 || lane == 3) edge[parity][warp][0][(lane - 2) * 2 + i] = x[i];
        if (lane == 28 || lane == 29) edge[parity][warp][1][(lane - 28) * 2 + i] = x[i];
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (lane < 2 && warp > 0) x[i] = edge[parity][warp - 1][1][lane * 2 + i];
        if (lane >= 30 && warp < kWarps - 1) x[i] = edge[parity][warp + 1][0][(lane - 30) * 2 + i];
      }
      parity ^= 1;
    }
    done += steps;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (mine[i]) {
      A[g[i]] = x[i];
      B[g[i]] = before[i];
    }
}

}  // namespace

// NPBGB_ERR_STATE (nothing launched; the caller then uses the chained launches) when
// the CTAs that fit one per SM cannot hold the array, when the launch is refused, or on a stream that is being
// captured (the chained launches need no scratch memory).
int32_t jacobi1d_resident_run(float* a, float* b, int64_t n, int32_t tsteps, cudaStream_t st) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone)
    return NPBGB_ERR_STATE;
  // Few CTAs with long halos where the array is small: a half-sweep takes the same time
  // in any span.  At least 32 half-sweeps a round (16: 1.43 ms, 32 1.11, 64 0.94, 120
  // 0.87 at N=32000).
  const int64_t w = std::max<int64_t>(cdiv(n - 2, sm_count()), 148);
  const int H = int(std::min<int64_t>((kSpan - w) / 2, w)) & ~3;
  if (H < 32 || tsteps > (1 << 30)) return NPBGB_ERR_STATE;  // (half-sweeps are counted in 32 bits)
  const int nb = int(cdiv(n - 2, w));
  const size_t bytes = size_t(4) * nb * size_t(H) * sizeof(Mail);
  cudaMemPool_t pool;
  void* scratch = nullptr;
  cudaError_t e;
  if ((e = scratch_pool(&pool)) != cudaSuccess ||
      (e = cudaMallocFromPoolAsync(&scratch, bytes, pool, st)) != cudaSuccess) {
    cudaGetLastError();
    return NPBGB_ERR_STATE;  // no memory for the mail
  }
  if (nb > 1) e = cudaMemsetAsync(scratch, 0, bytes, st);
  if (e == cudaSuccess) {
    auto* mail = static_cast<Mail*>(scratch);
    int hs = 2 * (tsteps - 1), w_ = int(w), H_ = H;
    void* args[] = {&a, &b, &n, &hs, &w_, &H_, &mail};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(nb));
    cfg.blockDim = dim3(32 * kWarps);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = launch_together(cfg, reinterpret_cast<const void*>(jacobi1d_resident), args);
  }
  cudaFreeAsync(scratch, st);
  return e == cudaSuccess ? NPBGB_OK : NPBGB_ERR_STATE;  // not launched
}

uint32_t take_jacobi1d_device_error() {
  unsigned int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_j1_error, sizeof(v)) != cudaSuccess) return 0xffffffffu;
  if (v) cudaMemcpyToSymbol(g_j1_error, &zero, sizeof(zero));
  return v;
}

}  // namespace npbgb
