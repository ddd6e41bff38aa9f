// Binary64 3D 7-point heat half-sweep in binary32 limbs (fxl.cuh); the point
// arithmetic and its order are heat3d.cu's.
//
// A CTA of 4 warps owns 8R x 32 points of the (axis 1, axis 2) plane and streams
// along axis 0.  Lane tx, warp ty owns R pairs of points: rows ty*R + r and
// ty*R + r + 4R of column tx, the two halves of each packed operation, so that
// every neighbour of a pair is the pair at the neighbouring row or column and no
// operand is ever re-paired.  Per plane a thread loads its pairs (plain coalesced
// loads one plane ahead, so any alignment), converts them once, keeps them in
// registers as this plane's axis-0 neighbour and the next plane's centre, and
// publishes them in shared memory for the in-plane neighbours; three warps also
// convert the tile's halo.  One CTA barrier per plane (three limb buffers).
//
// What bounds it: the packed binary32 pipe, 55 operations a point of 130
// instructions in all (ncu, 256^3), with 16 warps per SM.  One half-sweep of 256^3
// takes 92 us against 123 us for the integer form with hardware rows
// (heat3d_tma), 1.77e11 against 1.33e11 updates/s; rows of an odd length, which
// TMA cannot copy, 92 against 141 us at 255 x 253 x 251.  Tried and slower: 8
// warps per CTA (94 us), one pair per lane (99), three or four (110, 136), five
// CTAs per SM with a few spills (106), one wave of CTAs of equal length (99), an
// mbarrier per buffer instead of the CTA barrier (94), and hardware binary64 for
// one row in five or one tile in seven (121 and more: binary64 instructions
// stall the same dispatch).
//
// The limbs' range is [2^-7, 1), or that times a power of two which the CTA takes from
// the values at its tile's corners.  NPBench's initial field (values up to 20) then stays
// in limbs: TSTEPS=11 at 256^3 takes 2.2 ms, in hardware binary64 8.4 and in
// heat3d_tma 7.8; 25^3, TSTEPS=25, 0.16, 0.26 and 0.39.  Points whose inputs leave the
// range or whose result does (+0 is in it) are evaluated in hardware binary64 from
// global memory.
#include <cmath>

#include "fxl.cuh"
#include "heat_core.cuh"
#include "npbgb_common.cuh"

namespace npbgb {

extern int64_t g_cfg_heat_chunk;

namespace {

constexpr int kW = 4;      // warps per CTA
constexpr int kCols = 34;  // tile columns and one halo column on either side
template <int R>
constexpr int kCtas = R == 1 ? 7 : 4;  // CTAs per SM (72 and 120 registers a thread)

template <int W, int R>
struct Geom {
  static constexpr int kHalf = W * R;       // rows between the two points of a pair
  static constexpr int kTileRows = 2 * kHalf;
  static constexpr int kRows = kHalf + 2;    // pair rows with their halo
};

using fxl::L3;
using fxl::P2;

// One plane's limbs: h and m of a pair side by side, l apart.
template <int W, int R>
struct Plane {
  ulonglong2 hm[Geom<W, R>::kRows][kCols];
  unsigned long long l[Geom<W, R>::kRows][kCols];

  __device__ __forceinline__ void put(int r, int c, const L3& x) {
    hm[r][c] = make_ulonglong2(x.h.v, x.m.v);
    l[r][c] = x.l.v;
  }
  __device__ __forceinline__ L3 get(int r, int c) const {
    const ulonglong2 a = hm[r][c];
    return L3{P2{a.x}, P2{a.y}, P2{l[r][c]}};
  }
};

__device__ __forceinline__ uint64_t bits_of(double x) { return static_cast<uint64_t>(__double_as_longlong(x)); }

// 8 times one axis' term: (nx - 2c) + pv, both roundings.
__device__ __forceinline__ L3 axis(const fxl::Consts& K, const L3& c, const L3& nx, const L3& pv) {
  L3 s = fxl::fma(K.minus_two, c, nx);
  fxl::round_any(K, s);
  s = fxl::add(s, pv);
  fxl::round_any(K, s);
  return s;
}

// The point at q in hardware binary64; out of line, rarely taken.
__device__ __noinline__ double hardware_point(const double* q, int64_t s0, int64_t s1) {
  return hcore::heat_point<double>(q[0], q[s0], q[-s0], q[s1], q[-s1], q[1], q[-1]);
}

// A CTA's tile and chunk in hardware binary64.  The tile's columns are numbered along its
// rows, so that one which the array cuts short fills its warps all the same; a thread
// streams one in every 32 W of them, with in-plane neighbours from memory.  Bound by the
// binary64 pipe, nine operations a point, and the last wave of CTAs: standard normal
// values at 256^3, TSTEPS=11, 6.1 ms (the pipe alone 5.86), where limbs evaluated in
// vain first and points one by one took 6.8; two of the nine on the integer pipes
// (f64emu.cuh) 6.6.
template <int W, int R>
__device__ __noinline__ void run_hardware(const double* __restrict__ src, double* __restrict__ dst, int64_t n0,
                                          int64_t n1, int64_t n2, int chunk) {
  constexpr int kEach = 2 * R;
  const int64_t k0 = 1 + int64_t(blockIdx.x) * 32, j0 = 1 + int64_t(blockIdx.y) * Geom<W, R>::kTileRows;
  const int ib = 1 + int(blockIdx.z) * chunk;
  const int ie = ib + chunk < int(n0) - 1 ? ib + chunk : int(n0) - 1;
  const int columns = int(n2 - 1 - k0 < 32 ? n2 - 1 - k0 : 32);
  const int rows = int(n1 - 1 - j0 < Geom<W, R>::kTileRows ? n1 - 1 - j0 : Geom<W, R>::kTileRows);
  const int64_t s0 = n1 * n2;
  const double* p = src + int64_t(ib) * s0 + j0 * n2 + k0;
  double* o = dst + (p - src);
  const int first = int(threadIdx.x) & ~31;  // of the warp's columns
  const int points = rows * columns;
  uint32_t off[kEach];
  bool live[kEach];
  double before[kEach], at[kEach];
#pragma unroll
  for (int m = 0; m < kEach; ++m) {
    const int q = int(threadIdx.x) + m * 32 * W;
    live[m] = q < points;
    off[m] = live[m] ? uint32_t(q / columns) * uint32_t(n2) + uint32_t(q % columns) : 0u;
    before[m] = p[int64_t(off[m]) - s0];
    at[m] = p[off[m]];
  }
  for (int i = ib; i < ie; ++i) {
    double after[kEach], jp[kEach], jm[kEach], kp[kEach], km[kEach];
#pragma unroll
    for (int m = 0; m < kEach; ++m)
      if (first + m * 32 * W < points) {
        const double* c = p + off[m];
        after[m] = c[s0];
        jp[m] = c[n2];
        jm[m] = c[-n2];
        kp[m] = c[1];
        km[m] = c[-1];
      }
#pragma unroll
    for (int m = 0; m < kEach; ++m)
      if (first + m * 32 * W < points) {
        const double v = hcore::heat_point<double>(at[m], after[m], before[m], jp[m], jm[m], kp[m], km[m]);
        if (live[m]) o[off[m]] = v;
        before[m] = at[m];
        at[m] = after[m];
      }
    p += s0;
    o += s0;
  }
}

// A CTA's tile and chunk; 0 when it is done.  SCALED: in the frame that the values at the
// corners of its first plane (the same for every thread) ask for; with R = 2, not 0
// (nothing written) if three of four rows of pairs of that plane hold a value out of the
// frame, as nearly every warp would then evaluate its points twice.  Otherwise in the
// frame of zero, which costs no instructions, and not 0 (nothing written) if a centre
// pair of the first plane is out of range: bit 2 + r then says that one of the thread's
// pair r is negative.
template <int W, int R, bool SCALED>
__device__ __forceinline__ int run_chunk(const double* __restrict__ src, double* __restrict__ dst, int64_t n0,
                                         int64_t n1, int64_t n2, int chunk, Plane<W, R> (&plane)[3]) {
  using G = Geom<W, R>;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t k0 = 1 + int64_t(blockIdx.x) * 32, j0 = 1 + int64_t(blockIdx.y) * G::kTileRows;
  const int ib = 1 + int(blockIdx.z) * chunk;
  const int ie = ib + chunk < int(n0) - 1 ? ib + chunk : int(n0) - 1;
  const int64_t s0 = n1 * n2;
  const int64_t k = k0 + tx;
  const int row = ty * R;  // the first pair's row in the tile

  // Own points: in the array (loaded), in the interior (written).  Points
  // outside the array read as 0.5, a value that needs no second look.  Offsets within a plane are 32-bit bytes, next
  // to plane addresses that are the same for the whole grid.
  bool in_a[R], in_b[R], out_a[R], out_b[R];
  uint32_t off_a[R], off_b[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int64_t j = j0 + row + r;
    in_a[r] = k < n2 && j < n1;
    in_b[r] = k < n2 && j + G::kHalf < n1;
    out_a[r] = k < n2 - 1 && j < n1 - 1;
    out_b[r] = k < n2 - 1 && j + G::kHalf < n1 - 1;
    off_a[r] = uint32_t(j * n2 + k) * 8u;
    off_b[r] = uint32_t((j + G::kHalf) * n2 + k) * 8u;
  }
  auto ld = [](const double* plane_at, uint32_t off) {
    return *reinterpret_cast<const double*>(reinterpret_cast<const char*>(plane_at) + off);
  };
  struct Raw { double a, b; };
  auto load_own = [&](const double* p, Raw (&x)[R]) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      x[r].a = in_a[r] ? ld(p, off_a[r]) : 0.5;
      x[r].b = in_b[r] ? ld(p, off_b[r]) : 0.5;
    }
  };
  // The halo of a plane: pair row 0 (the row before the tile and the last row of
  // its first half; warp 0), pair row kRows-1 (warp 1), and the two halo
  // columns (warp 2).
  int hr = -1, hc = tx + 1;
  if (ty == 0) hr = 0;
  else if (ty == 1) hr = G::kRows - 1;
  else if (ty == 2 && tx < 2 * G::kHalf) {
    hr = 1 + tx % G::kHalf;
    hc = tx < G::kHalf ? 0 : kCols - 1;
  }
  const int64_t hk = k0 - 1 + hc, hj = j0 + hr - 1;
  const bool hin_a = hr >= 0 && hk < n2 && hj < n1;
  const bool hin_b = hr >= 0 && hk < n2 && hj + G::kHalf < n1;
  const uint32_t hoff_a = uint32_t(hj * n2 + hk) * 8u, hoff_b = uint32_t((hj + G::kHalf) * n2 + hk) * 8u;
  auto load_halo = [&](const double* p, Raw& x) {
    x.a = hin_a ? ld(p, hoff_a) : 0.5;
    x.b = hin_b ? ld(p, hoff_b) : 0.5;
  };

  fxl::Consts K = fxl::consts();
  auto limbs = [&](const Raw& x) { return fxl::from_f64(K, bits_of(x.a), bits_of(x.b)); };
  Raw own[R], halo{0.5, 0.5};
  L3 x0[R], x1[R], x2[R];
  const double* p = src + int64_t(ib - 1) * s0;
  load_own(p, own);
  uint32_t corner[4] = {0u, 0u, 0u, 0u};
  if (SCALED) {
    const uint32_t last_j = uint32_t((j0 + G::kTileRows < n1 ? j0 + G::kTileRows : n1) - 1 - j0) * uint32_t(n2);
    const uint32_t last_k = uint32_t((k0 + 32 < n2 ? k0 + 32 : n2) - 1 - k0);
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p + s0 + j0 * n2 + k0) + 1;  // upper words
    corner[0] = q[0];
    corner[1] = q[2 * last_k];
    corner[2] = q[2 * last_j];
    corner[3] = q[2 * (last_j + last_k)];
  }
  Raw own1[R];
  p += s0;
  load_own(p, own1);
  if (hr >= 0) load_halo(p, halo);
  if (SCALED) {
    uint32_t top = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) top = corner[c] < 0x7ff00000u && corner[c] > top ? corner[c] : top;
    K.scale = fxl::frame_of(top);
  }
  if (SCALED && R == 2) {
    bool counts = false;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool a = in_a[r] && fxl::refused(K, bits_of(own1[r].a)), b = in_b[r] && fxl::refused(K, bits_of(own1[r].b));
      if (__any_sync(0xffffffffu, a || b) && tx == r) counts = true;
    }
    if (__syncthreads_count(counts) * 4 >= 3 * W * R) return 1;
  }
#pragma unroll
  for (int r = 0; r < R; ++r) x0[r] = limbs(own[r]);
  bool out_of_range = false;
  uint32_t negative = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (!SCALED && int((bits_of(own1[r].a) | bits_of(own1[r].b)) >> 32) < 0) negative |= 4u << r;
    x1[r] = limbs(own1[r]);
    out_of_range = out_of_range || fxl::refused_both(x1[r]);
    plane[0].put(row + r + 1, tx + 1, x1[r]);
  }
  if (hr >= 0) plane[0].put(hr, hc, limbs(halo));
  p += s0;
  load_own(p, own);
  if (hr >= 0 && ib + 1 < ie) load_halo(p, halo);
  if (SCALED)
    __syncthreads();
  else if (__syncthreads_or(out_of_range))
    return int(1u | negative);

  double* o = dst + int64_t(ib) * s0;
  int i = ib;
  // Output plane i from planes i - 1 (im), i (c, published in `now`) and i + 1,
  // which it converts into ip and publishes in `next`, loading plane i + 2.
  // False after the last plane.
  auto step = [&](const L3 (&im)[R], const L3 (&c)[R], L3 (&ip)[R], int bn) -> bool {
    const Plane<W, R>& now = plane[bn];
    Plane<W, R>& next = plane[bn == 2 ? 0 : bn + 1];
#pragma unroll
    for (int r = 0; r < R; ++r) ip[r] = limbs(own[r]);
    if (i + 1 < ie) {
#pragma unroll
      for (int r = 0; r < R; ++r) next.put(row + r + 1, tx + 1, ip[r]);
      if (hr >= 0) next.put(hr, hc, limbs(halo));
      p += s0;
      load_own(p, own);
      if (hr >= 0 && i + 2 < ie) load_halo(p, halo);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int pr = row + r + 1;
      const L3 jm = r > 0 ? c[r > 0 ? r - 1 : 0] : now.get(pr - 1, tx + 1);
      const L3 jp = r + 1 < R ? c[r + 1 < R ? r + 1 : r] : now.get(pr + 1, tx + 1);
      L3 w = axis(K, c[r], ip[r], im[r]);
      w = fxl::add(w, axis(K, c[r], jp, jm));
      fxl::round_any(K, w);
      w = fxl::add(w, axis(K, c[r], now.get(pr, tx + 2), now.get(pr, tx)));
      fxl::round_any(K, w);
      w = fxl::fma(K.eight, c[r], w);
      const P2 e = fxl::round_any(K, w);
      const fxl::Words q = fxl::words_of(K, w);
      double va = __longlong_as_double(
          fxl::to_f64<62>(fxl::first(q.h), fxl::first(q.m), fxl::first(q.l), fxl::first(e), K.scale));
      double vb = __longlong_as_double(
          fxl::to_f64<62>(fxl::second(q.h), fxl::second(q.m), fxl::second(q.l), fxl::second(e), K.scale));
      if (!(fxl::within<-4, 3>(fxl::first(e)) && fxl::within<-4, 3>(fxl::second(e)))) {
        const double* g = src + (o - dst);
        // All inputs of a sum of nothing (e = 0) were in limbs: it is +0.  Evaluated in
        // hardware, a field of zeros took 9.0 ms at 256^3, TSTEPS=11, instead of 2.0.
        if (!fxl::within<-4, 3>(fxl::first(e)))
          va = out_a[r] && fxl::first(e) != 0u ? hardware_point(g + off_a[r] / 8, s0, n2) : 0.0;
        if (!fxl::within<-4, 3>(fxl::second(e)))
          vb = out_b[r] && fxl::second(e) != 0u ? hardware_point(g + off_b[r] / 8, s0, n2) : 0.0;
      }
      if (out_a[r]) *reinterpret_cast<double*>(reinterpret_cast<char*>(o) + off_a[r]) = va;
      if (out_b[r]) *reinterpret_cast<double*>(reinterpret_cast<char*>(o) + off_b[r]) = vb;
    }
    o += s0;
    ++i;
    __syncthreads();
    return i < ie;
  };
  // The register sets and buffers change roles by unrolling, without moves.
  while (step(x0, x1, x2, 0) && step(x1, x2, x0, 1) && step(x2, x0, x1, 2)) {
  }
  return 0;
}

// Out of line, so that the kernel's registers are the other form's.  Bit r of `negative`:
// one of the thread's pair r is negative, which no frame holds.
template <int W, int R>
__device__ __noinline__ void run_scaled(const double* __restrict__ src, double* __restrict__ dst, int64_t n0,
                                        int64_t n1, int64_t n2, int chunk, uint32_t negative,
                                        Plane<W, R> (&plane)[3]) {
  bool counts = false;
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (__any_sync(0xffffffffu, (negative >> r) & 1u) && int(threadIdx.x & 31) == r) counts = true;
  if (__syncthreads_count(counts) * 4 >= 3 * W * R || run_chunk<W, R, true>(src, dst, n0, n1, n2, chunk, plane))
    run_hardware<W, R>(src, dst, n0, n1, n2, chunk);
}

// With two pairs a thread a CTA tries the frame of zero first: the scale in every
// conversion costs 3.5% at 256^3.  With one pair that form needs more registers than
// seven CTAs per SM leave (120^3: 0.605 ms against 0.593, and 0.58 without any scale), and
// so does run_hardware (130^3, TSTEPS=21: 0.733 ms against 0.707, for 1.68 against 1.71
// on standard normal values).
template <int W, int R>
__global__ void __launch_bounds__(32 * W, kCtas<R>)
heat3d_limb(const double* __restrict__ src, double* __restrict__ dst, int64_t n0, int64_t n1,
            int64_t n2, int chunk) {
  pdl_begin();
  __shared__ Plane<W, R> plane[3];
  if constexpr (R == 1) {
    run_chunk<W, R, true>(src, dst, n0, n1, n2, chunk, plane);
  } else if (const int how = run_chunk<W, R, false>(src, dst, n0, n1, n2, chunk, plane)) {
    run_scaled<W, R>(src, dst, n0, n1, n2, chunk, uint32_t(how) >> 2, plane);
  }
}

template <int R>
int32_t launch(double* a, double* b, int64_t n0, int64_t n1, int64_t n2, int32_t tsteps, int chunk,
               cudaStream_t st) {
  const dim3 grid{unsigned(cdiv(n2 - 2, 32)), unsigned(cdiv(n1 - 2, Geom<kW, R>::kTileRows)),
                  unsigned(cdiv(n0 - 2, chunk))};
  cudaError_t e = cudaSuccess;
  for (int32_t t = 1; t < tsteps && e == cudaSuccess; ++t) {
    e = launch_chained(heat3d_limb<kW, R>, grid, dim3{32u * kW}, 0, st, a, b, n0, n1, n2, chunk);
    if (e == cudaSuccess)
      e = launch_chained(heat3d_limb<kW, R>, grid, dim3{32u * kW}, 0, st, b, a, n0, n1, n2, chunk);
  }
  return cuda_status(e, "heat3d_limb");
}

// The form for a grid.  q counts the planes of a tile (units) per CTA that the
// GPU holds at once.  Two pairs per lane (R = 2) convert fewer halo values and
// share axis-1 neighbours, one (R = 1) has smaller tiles: measured on GB300 at
// TSTEPS=21, 256^3 3.68 ms with R = 2 and 3.93 with R = 1, 120^3 0.62 / 0.61,
// 70^3 0.30 / 0.28.  The planes per CTA follow 1.45 sqrt(q): few CTAs with long
// chunks waste fewer halo planes, many short ones balance the last wave.
// Measured best: 1 plane at q = 0.6 (48^3: 0.186 ms; 2 planes 0.233), 2 at q = 2
// (70^3: 0.282; 1 0.294, 4 0.356), 4 at q = 8 (120^3: 0.605; 8 0.677), 10 to 12 at
// q = 53 (256^3: 3.68; 4 4.04, 20 3.77).
template <int R>
double planes_per_slot(int64_t n0, int64_t n1, int64_t n2) {
  const int64_t units = cdiv(n2 - 2, 32) * cdiv(n1 - 2, Geom<kW, R>::kTileRows) * (n0 - 2);
  return double(units) / double(int64_t(sm_count()) * kCtas<R>);
}

}  // namespace

// NPBGB_ERR_STATE (nothing launched) when a plane exceeds the kernel's 32-bit
// offsets or a grid dimension is too large.
int32_t heat3d_limb_run(double* a, double* b, int64_t n0, int64_t n1, int64_t n2, int32_t tsteps,
                        cudaStream_t st) {
  if (n1 > 0x7fffffff || n2 > 0x7fffffff || n1 * n2 >= (int64_t(1) << 29) || n0 > 0x7fffffff)
    return NPBGB_ERR_STATE;
  const bool two = planes_per_slot<2>(n0, n1, n2) >= 12.0;
  const double q = two ? planes_per_slot<2>(n0, n1, n2) : planes_per_slot<1>(n0, n1, n2);
  int64_t chunk = g_cfg_heat_chunk > 0 ? g_cfg_heat_chunk : int64_t(1.45 * std::sqrt(q) + 0.5);
  if (chunk < 1) chunk = 1;
  if (chunk > n0 - 2) chunk = n0 - 2;
  if (cdiv(n0 - 2, chunk) > 65535 || cdiv(n1 - 2, Geom<kW, 1>::kTileRows) > 65535)
    return NPBGB_ERR_STATE;
  return two ? launch<2>(a, b, n0, n1, n2, tsteps, int(chunk), st)
             : launch<1>(a, b, n0, n1, n2, tsteps, int(chunk), st);
}

}  // namespace npbgb
