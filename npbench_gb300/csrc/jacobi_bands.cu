// Jacobi-2D with the whole time loop in one launch: bands resident in shared memory.
//
// For grids that shared memory holds, chained launches spend most of a half-sweep on launch ramp-up, short row chunks and L2
// latency.  Here one cooperative launch runs all 2*(TSTEPS-1) half-sweeps of
// polybench/jacobi_2d/jacobi_2d_numpy.py:6-10.  CTA b owns a band of R interior
// rows; a thread owns CPT adjacent columns of it for the whole run.
//
//   * Rows i and i + H of a column (H = ceil(R/2)) are the two
//     halves of one packed operand, pair i of 0 .. H-1, so every neighbour of a pair is
//     a pair.  A thread's columns lie in shared memory that only it touches, in one
//     copy: a half-sweep walks along them with three pairs of the old field in
//     registers and writes each new pair over the old one.  The three are moved from
//     step to step: with the loop unrolled by three instead, so that only names move,
//     the point code is six times in the kernel and fetching it cost more (binary64
//     1000^2: 8.5 against 7.4 us a half-sweep).
//   * West and east neighbours come from the thread's other columns and by shuffle;
//     only the outer columns of each warp are shared with other warps (one CTA barrier
//     per half-sweep, two buffers).
//   * Bands of one thread-block cluster pass edge values straight into each other's
//     shared memory (st.async, counted by an mbarrier there).  Across clusters an
//     edge value travels through L2 as one tagged element ({value, sweep} as 64 bits,
//     or three limbs and the sweep as 128) that is stored with a single-copy-atomic
//     access; extra warps poll for such elements and put them into shared memory
//     behind the same mbarrier, so no thread that computes waits for a load.
//     Even half-sweeps walk down and odd ones up: the edge sent first is the one that
//     the neighbour needs first in its next half-sweep, and the one sent last is
//     needed last, so the trip hides behind the arithmetic both ways.
//   * Faces: column 0 and nx-1 and the first and last rows hold A's values in even
//     fields and B's in odd ones, as in the reference's arrays.  The last
//     half-sweep's input goes to B and its result to A.
//
// binary32 points are five packed operations.  binary64 cells are kept as three
// binary32 limbs (fxl.cuh) for all half-sweeps, the product by 0.2 included; a cell
// outside their range holds NaN and the value's own bits in the other two words,
// and a point that touches one is evaluated in hardware binary64.
//
// Bound by the instructions of a point and by the hand-off's latency: a half-sweep of
// binary32 1403 x 1177 takes 2.2 us where the points alone take about 1.5.  Measured,
// chained launches to bands, TSTEPS=100: binary32 1000^2 0.72 to 0.40 ms, 1403 x 1177
// 1.02 to 0.48, 2048^2 (TSTEPS=50) 0.785 to 0.39; binary64 on values in [0, 1) 300^2 (50)
// 0.30 to 0.25.  With every edge through L2 the 1403 x 1177 grid took 0.85 ms,
// with the computing threads polling instead of extra warps 0.71.
//
// Places of edge values alternate between two slots.  A thread sends sweep s+1 of a
// column over s-1 after it has taken sweep s of that column from the same neighbour,
// whose thread sent it after it had taken s-1; so the place of s-1 is free by then.
// Every wait is bounded: a neighbour that sends nothing for seconds sets an error
// word, the band stops waiting, and all bands of the cluster leave together.
//
// Mail and halos are laid out for the cluster size that the host asked for.  A launch
// that runs in other clusters (Nsight Compute launches a cooperative kernel's CTAs one
// by one) is told by the hardware's own count and takes in_memory instead.
#include <algorithm>
#include <atomic>
#include <type_traits>
#include <mutex>

#include "fxl.cuh"
#include "npbgb_common.cuh"
#include "tma.cuh"

namespace npbgb {

extern int64_t g_cfg_f64_emulation;
extern int64_t g_cfg_jacobi_bands;

namespace {

constexpr uint64_t kJLimitNs = 2000000000ull;

__device__ unsigned int g_jbands_error;  // bit 0: a neighbour wait gave up

using fxl::L3;
using fxl::P2;

// ---------------------------------------------------------------------------
// Cells: one value (Cell), two (Pair), their storage and their arithmetic
// ---------------------------------------------------------------------------
template <typename T>
struct Kind;

__device__ __forceinline__ P2 shfl_up1(P2 a) {
  return fxl::pair(__shfl_up_sync(0xffffffffu, fxl::first(a), 1), __shfl_up_sync(0xffffffffu, fxl::second(a), 1));
}
__device__ __forceinline__ P2 shfl_down1(P2 a) {
  return fxl::pair(__shfl_down_sync(0xffffffffu, fxl::first(a), 1),
                   __shfl_down_sync(0xffffffffu, fxl::second(a), 1));
}

// Into the shared memory of a CTA of the cluster, counted by its mbarrier `bar`.
__device__ __forceinline__ void send2(uint32_t to, uint32_t bar, uint32_t a, uint32_t b) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(to), "r"(a),
               "r"(b), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void send4(uint32_t to, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to),
               "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar)
               : "memory");
}

template <>
struct Kind<float> {
  struct Cell { uint32_t v; };
  using Pair = P2;
  struct Consts { P2 fifth; };
  using Mail = unsigned long long;
  static constexpr int kPairBytes = 8;
  static __device__ __forceinline__ Consts consts() { return Consts{fxl::opaque_both(__float_as_uint(0.2f))}; }

  // Pairs in shared memory, addressed by 32-bit offsets of slots (one pair each).
  struct Store {
    unsigned long long* x;
    __device__ __forceinline__ Store(unsigned char* at, int) : x(reinterpret_cast<unsigned long long*>(at)) {}
    __device__ __forceinline__ Pair get(int i) const { return Pair{x[i]}; }
    __device__ __forceinline__ void put(int i, Pair v) const { x[i] = v.v; }
    __device__ __forceinline__ void put_half(int i, int which, Cell v) const {
      reinterpret_cast<uint32_t*>(x + i)[which] = v.v;
    }
  };
  static __device__ __forceinline__ Pair select(bool c, Pair a, Pair b) { return Pair{c ? a.v : b.v}; }
  static __device__ __forceinline__ Pair up1(Pair v) { return shfl_up1(v); }
  static __device__ __forceinline__ Pair down1(Pair v) { return shfl_down1(v); }
  static __device__ __forceinline__ Cell half(Pair v, int which) {
    return Cell{which ? fxl::second(v) : fxl::first(v)};
  }
  static __device__ __forceinline__ Pair join(Cell a, Cell b) { return fxl::pair(a.v, b.v); }
  static __device__ __forceinline__ Cell cell(const Consts&, float v) { return Cell{__float_as_uint(v)}; }
  static __device__ __forceinline__ float value(Cell c) { return __uint_as_float(c.v); }
  struct Work {};
  static __device__ __forceinline__ Pair point(const Consts& k, const Pair& c, const Pair& w, const Pair& e,
                                               const Pair& s, const Pair& n, Work&) {
    const P2 sum = fxl::add(fxl::add(fxl::add(fxl::add(c, w), e), s), n);
    return P2{mul2(F2{k.fifth.v}, F2{sum.v}).v};
  }
  static __device__ __forceinline__ bool sure(const Work&, bool, bool) { return true; }
  static __device__ __forceinline__ Pair mend(Pair r, const Work&, bool, bool, const Pair&, const Pair&, const Pair&,
                                              const Pair&, const Pair&) {
    return r;
  }
  // Halo rows: a thread's columns adjacent, so that they travel together.
  using Halo = uint32_t;
  template <int CPT>
  static __device__ __forceinline__ int halo_index(int c, int thread, int) { return thread * CPT + c; }
  static __device__ __forceinline__ Cell cell(Halo h) { return Cell{h}; }
  static __device__ __forceinline__ Halo halo(Cell c) { return c.v; }
  template <int CPT>
  static __device__ __forceinline__ void send(uint32_t to, uint32_t bar, int thread, int, const Cell (&v)[CPT]) {
    to += thread * CPT * 4;
    if constexpr (CPT == 2) {
      send2(to, bar, v[0].v, v[1].v);
    } else {
#pragma unroll
      for (int c = 0; c < CPT; c += 4) send4(to + c * 4, bar, v[c].v, v[c + 1].v, v[c + 2].v, v[c + 3].v);
    }
  }
  template <int CPT>
  static __device__ __forceinline__ void post(Mail* box, uint32_t tag, int thread, int, const Cell (&v)[CPT]) {
    const unsigned long long t = static_cast<unsigned long long>(tag) << 32;
#pragma unroll
    for (int c = 0; c < CPT; c += 2)
      asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(box + thread * CPT + c), "l"(t | v[c].v),
                   "l"(t | v[c + 1].v)
                   : "memory");
  }
  // A mailbox element as loaded; its tag is looked at later.
  struct Letter { unsigned long long x; };
  static __device__ __forceinline__ Letter peek(const Mail* at) {
    Letter r;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(r.x) : "l"(at) : "memory");
    return r;
  }
  static __device__ __forceinline__ Cell cell(const Letter& r) { return Cell{static_cast<uint32_t>(r.x)}; }
  static __device__ __forceinline__ uint32_t tag(const Letter& r) { return static_cast<uint32_t>(r.x >> 32); }
};

template <>
struct Kind<double> {
  struct Cell { uint32_t h, m, l; };
  using Pair = L3;
  using Consts = fxl::Consts;
  using Mail = ulonglong2;
  static constexpr int kPairBytes = 24;
  static __device__ __forceinline__ Consts consts() { return fxl::consts(); }

  struct Store {
    ulonglong2* hm;
    unsigned long long* l;
    __device__ __forceinline__ Store(unsigned char* at, int slots)
        : hm(reinterpret_cast<ulonglong2*>(at)), l(reinterpret_cast<unsigned long long*>(at + size_t(slots) * 16)) {}
    __device__ __forceinline__ Pair get(int i) const {
      const ulonglong2 a = hm[i];
      return L3{P2{a.x}, P2{a.y}, P2{l[i]}};
    }
    __device__ __forceinline__ void put(int i, const Pair& v) const {
      hm[i] = make_ulonglong2(v.h.v, v.m.v);
      l[i] = v.l.v;
    }
    __device__ __forceinline__ void put_half(int i, int which, Cell v) const {
      uint32_t* q = reinterpret_cast<uint32_t*>(hm + i);
      q[which] = v.h;
      q[2 + which] = v.m;
      reinterpret_cast<uint32_t*>(l + i)[which] = v.l;
    }
  };
  static __device__ __forceinline__ Pair select(bool c, const Pair& a, const Pair& b) {
    return L3{P2{c ? a.h.v : b.h.v}, P2{c ? a.m.v : b.m.v}, P2{c ? a.l.v : b.l.v}};
  }
  static __device__ __forceinline__ Pair up1(const Pair& v) { return L3{shfl_up1(v.h), shfl_up1(v.m), shfl_up1(v.l)}; }
  static __device__ __forceinline__ Pair down1(const Pair& v) {
    return L3{shfl_down1(v.h), shfl_down1(v.m), shfl_down1(v.l)};
  }
  static __device__ __forceinline__ Cell half(const Pair& v, int which) {
    return which ? Cell{fxl::second(v.h), fxl::second(v.m), fxl::second(v.l)}
                 : Cell{fxl::first(v.h), fxl::first(v.m), fxl::first(v.l)};
  }
  static __device__ __forceinline__ Pair join(Cell a, Cell b) {
    return L3{fxl::pair(a.h, b.h), fxl::pair(a.m, b.m), fxl::pair(a.l, b.l)};
  }
  // Limbs, or NaN and the value's own bits.
  static __device__ __forceinline__ Cell cell(const Consts& k, double v) {
    const uint64_t b = static_cast<uint64_t>(__double_as_longlong(v));
    const L3 x = fxl::from_f64(k, b, b);
    if (!fxl::refused_value(x)) return half(x, 0);
    return Cell{fxl::kNaN, static_cast<uint32_t>(b >> 32), static_cast<uint32_t>(b)};
  }
  static __device__ double value(Cell c) {
    if (c.h == fxl::kNaN)
      return __longlong_as_double(static_cast<long long>(static_cast<uint64_t>(c.m) << 32 | c.l));
    const Consts k = fxl::consts();
    const fxl::Words w = fxl::words_of(k, join(c, c));
    return fx::to_f64<59>(fxl::to_fx(fxl::first(w.h), fxl::first(w.m), fxl::first(w.l)));
  }
  static __device__ __noinline__ Cell hardware(Cell c, Cell w, Cell e, Cell s, Cell n) {
    double acc = add_rn(value(c), value(w));
    acc = add_rn(acc, value(e));
    acc = add_rn(acc, value(s));
    acc = add_rn(acc, value(n));
    return cell(fxl::consts(), mul_rn(0.2, acc));
  }
  // 0.2 times a rounded sum (53 significant bits, so both additions are exact).
  static __device__ __noinline__ Cell fifth_hardware(Cell s) {
    const double hm = add_rn(double(__uint_as_float(s.h)), double(__uint_as_float(s.m)));
    const double l = mul_rn(double(__uint_as_float(s.l)), 0x1p-29);
    return cell(fxl::consts(), mul_rn(0.2, mul_rn(add_rn(hm, l), 0x1p-8)));
  }
  // What a point leaves open: its rounded sum, and which products stand.
  struct Work {
    L3 x;
    P2 t;
    bool a, b;
  };
  static __device__ __forceinline__ Pair point(const Consts& k, const Pair& c, const Pair& w, const Pair& e,
                                               const Pair& s, const Pair& n, Work& o) {
    o.x = fxl::add(c, w);
    fxl::round_pos(k, o.x);
    o.x = fxl::add(o.x, e);
    fxl::round_pos(k, o.x);
    o.x = fxl::add(o.x, s);
    fxl::round_pos(k, o.x);
    o.x = fxl::add(o.x, n);
    fxl::round_pos(k, o.x, o.t);
    return fxl::fifth_of(k, o.x, o.t, o.a, o.b);
  }
  static __device__ __forceinline__ bool sure(const Work& o, bool need_a, bool need_b) {
    return (o.a || !need_a) && (o.b || !need_b);
  }
  // The products that are open: zero sums are zero, ties and powers of two take the
  // hardware's product, and sums with a value out of range the hardware altogether.
  struct Point {
    Pair c, w, e, s, n, r;
    Work o;
  };
  static __device__ __noinline__ void mend_point(Point& q, bool need_a, bool need_b) {
    auto other = [&](uint32_t t, int which) {
      if (t == 0u) return Cell{0u, 0u, 0u};
      if ((t << 1) <= 0xff000000u) return fifth_hardware(half(q.o.x, which));
      return hardware(half(q.c, which), half(q.w, which), half(q.e, which), half(q.s, which), half(q.n, which));
    };
    const Cell a = q.o.a || !need_a ? half(q.r, 0) : other(fxl::first(q.o.t), 0);
    const Cell b = q.o.b || !need_b ? half(q.r, 1) : other(fxl::second(q.o.t), 1);
    q.r = join(a, b);
  }
  static __device__ __forceinline__ Pair mend(const Pair& r, const Work& o, bool need_a, bool need_b, const Pair& c,
                                              const Pair& w, const Pair& e, const Pair& s, const Pair& n) {
    Point q{c, w, e, s, n, r, o};
    mend_point(q, need_a, need_b);
    return q.r;
  }
  using Halo = uint4;
  template <int CPT>
  static __device__ __forceinline__ int halo_index(int c, int thread, int threads) { return c * threads + thread; }
  static __device__ __forceinline__ Cell cell(const Halo& h) { return Cell{h.x, h.y, h.z}; }
  static __device__ __forceinline__ Halo halo(Cell c) { return make_uint4(c.h, c.m, c.l, 0u); }
  template <int CPT>
  static __device__ __forceinline__ void send(uint32_t to, uint32_t bar, int thread, int threads,
                                              const Cell (&v)[CPT]) {
#pragma unroll
    for (int c = 0; c < CPT; ++c) send4(to + (c * threads + thread) * 16, bar, v[c].h, v[c].m, v[c].l, 0u);
  }
  template <int CPT>
  static __device__ __forceinline__ void post(Mail* box, uint32_t tag, int thread, int threads,
                                              const Cell (&v)[CPT]) {
#pragma unroll
    for (int c = 0; c < CPT; ++c)
      asm volatile("{\n.reg .b128 q;\nmov.b128 q, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], q;\n}" ::"l"(
                       box + c * threads + thread),
                   "l"(static_cast<unsigned long long>(v[c].m) << 32 | v[c].h),
                   "l"(static_cast<unsigned long long>(tag) << 32 | v[c].l)
                   : "memory");
  }
  struct Letter { unsigned long long x, y; };
  static __device__ __forceinline__ Letter peek(const Mail* at) {
    Letter r;
    asm volatile("{\n.reg .b128 q;\nld.relaxed.gpu.global.b128 q, [%2];\nmov.b128 {%0, %1}, q;\n}"
                 : "=l"(r.x), "=l"(r.y)
                 : "l"(at)
                 : "memory");
    return r;
  }
  static __device__ __forceinline__ Cell cell(const Letter& r) {
    return Cell{static_cast<uint32_t>(r.x), static_cast<uint32_t>(r.x >> 32), static_cast<uint32_t>(r.y)};
  }
  static __device__ __forceinline__ uint32_t tag(const Letter& r) { return static_cast<uint32_t>(r.y >> 32); }
};

// ---------------------------------------------------------------------------
// The kernel
// ---------------------------------------------------------------------------
// Threads that compute, at most, and warps that poll.
template <typename T>
constexpr int kPollWarps = sizeof(T) == 8 ? 1 : 4;
template <typename T, int CPT>
constexpr int kCompute = sizeof(T) == 4 ? 512 : CPT == 3 ? 352 : 480;

// A barrier of the computing threads alone; whether any of them said so.
__device__ __forceinline__ bool compute_sync_or(int threads, bool v) {
  uint32_t r;
  asm volatile(
      "{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbarrier.cta.red.or.pred q, 1, %2, p;\nselp.u32 %0, 1, 0, q;\n}"
      : "=r"(r)
      : "r"(v ? 1u : 0u), "r"(threads)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tma::smem_u32(bar)) : "memory");
}
// Waits for a phase that other CTAs of the cluster complete; false past the limit.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, uint64_t limit_ns) {
  uint64_t t0 = 0;
  for (uint32_t n = 1;; ++n) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(tma::smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
    if ((n & 63u) == 0) {
      const uint64_t now = tma::globaltimer();
      if (t0 == 0) t0 = now;
      if (now - t0 > limit_ns) return false;
    }
  }
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t in_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// Shared memory of a band: the mbarriers, the halo rows ([above, below][parity]), which
// are at the same place in every band, and slots of one pair.  Row p of the field
// holds the threads' columns ([c][thread]) and column nx-1 of both fields (A's, B's);
// then come the warps' outer columns.
template <typename T, int CPT>
struct Layout {
  static constexpr int kWarps = kCompute<T, CPT> / 32;
  int row, edge, slots;
  size_t halo, field, total;
  __host__ __device__ Layout(int H, int threads) {
    row = CPT * threads + 2;
    edge = H * row;
    // [parity][west, east of warp -1 .. kWarps][p]; the outermost are written and never read
    slots = edge + 2 * 2 * (kWarps + 2) * H;
    halo = 4 * sizeof(uint64_t);
    field = halo + size_t(4) * CPT * threads * sizeof(typename Kind<T>::Halo);
    total = field + size_t(slots) * Kind<T>::kPairBytes;
  }
};

// Bands have base or base + 1 rows, the longer ones first.
template <typename T, int CPT>
__device__ __forceinline__ void run_band(T* __restrict__ A, T* __restrict__ B, int ny, int nx, int halfsweeps,
                                         int base, int extra, int nb, typename Kind<T>::Mail* __restrict__ mail) {
  using K = Kind<T>;
  using Cell = typename K::Cell;
  using Pair = typename K::Pair;
  extern __shared__ __align__(16) unsigned char smem[];
  const int nt = blockDim.x - 32 * kPollWarps<T>;  // computing threads
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b = blockIdx.x;
  uint32_t rank, in_cluster;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(in_cluster));
  const int R = base + (b < extra ? 1 : 0), H = (R + 1) >> 1;
  const Layout<T, CPT> lay(H, nt);
  const typename K::Store store(smem + lay.field, lay.slots);
  typename K::Halo* const halo = reinterpret_cast<typename K::Halo*>(smem + lay.halo);
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smem);  // [above, below][parity]
  const typename K::Consts k = K::consts();
  const int r0 = 1 + b * base + (b < extra ? b : extra);
  const bool lowest = b == 0, highest = b == nb - 1;
  const int columns = CPT * nt;
  // A side (0 above, 1 below) is a wall, a band of this cluster, or one of another.
  auto wall = [&](int which) { return which ? highest : lowest; };
  auto near = [&](int which) { return which ? rank + 1 < in_cluster && !highest : rank > 0; };

  // Elements between clusters q and q + 1: downward (0) and upward (1), per parity.
  // Elements lie in a halo row's order, and every band cuts its columns alike.
  auto box = [&](int which, int dir, uint32_t tag) {
    const int q = b / int(in_cluster) - (which ? 0 : 1);
    return mail + (int64_t(q * 2 + dir) * 2 + int64_t(tag & 1u)) * columns;
  };
  auto halo_at = [&](int which, int s) { return halo + (which * 2 + (s & 1)) * columns; };
  if (tid == 0) {
    for (int q = 0; q < 4; ++q) {
      tma::mbar_init(&bars[q], near(q >> 1) ? 1 : kPollWarps<T>);
      // Fields 1 and 2; field s + 2 is announced when field s has been taken.
      if (near(q >> 1)) tma::mbar_arrive_expect_tx(&bars[q], columns * sizeof(typename K::Halo));
    }
    tma::fence_mbar_init();
  }
  // Halo rows of field 0 (A's rows); a wall's of both fields, for good.
  for (int q = tid; q < 2 * columns; q += blockDim.x) {
    const int which = q / columns, c = q % columns / nt, t = q % nt;
    const int j = 1 + t * CPT + c < nx ? 1 + t * CPT + c : nx - 1;
    const int64_t at = int64_t(which ? r0 + R : r0 - 1) * nx + j;
    const int i = K::template halo_index<CPT>(c, t, nt);
    halo_at(which, 0)[i] = K::halo(K::cell(k, __ldcg(A + at)));
    if (wall(which)) halo_at(which, 1)[i] = K::halo(K::cell(k, __ldcg(B + at)));
  }
  cluster_sync();  // no value is sent before the barriers stand

  if (tid >= nt) {
    // Polling warps: a band has at most one side towards another cluster.
    __syncthreads();
    __syncthreads();
    const int which = !wall(0) && !near(0) ? 0 : 1;
    if (wall(which) || near(which)) return;
    constexpr int kStride = 32 * kPollWarps<T>;
    auto poll = [&](auto at_once) {
      constexpr int kAtOnce = decltype(at_once)::value;
      for (int s = 1; s < halfsweeps; ++s) {
        const typename K::Mail* from = box(which, which, uint32_t(s));
        typename K::Halo* to = halo_at(which, s);
        bool ok = true;
        for (int e0 = tid - nt; e0 - lane < columns; e0 += kStride * kAtOnce) {
          bool need[kAtOnce];
#pragma unroll
          for (int m = 0; m < kAtOnce; ++m) need[m] = e0 + kStride * m < columns;
          uint64_t t0 = 0;
          for (uint32_t n = 1; ok; ++n) {
            typename K::Letter got[kAtOnce];
#pragma unroll
            for (int m = 0; m < kAtOnce; ++m)
              if (need[m]) got[m] = K::peek(from + e0 + kStride * m);
            bool missing = false;
#pragma unroll
            for (int m = 0; m < kAtOnce; ++m)
              if (need[m]) {
                if (K::tag(got[m]) == uint32_t(s)) {
                  to[e0 + kStride * m] = K::halo(K::cell(got[m]));
                  need[m] = false;
                } else {
                  missing = true;
                }
              }
            if (!missing) break;
            if ((n & 255u) == 0) {
              const uint64_t now = tma::globaltimer();
              if (t0 == 0) t0 = now;
              if (now - t0 > kJLimitNs) {
                atomicOr(&g_jbands_error, 1u);
                ok = false;
              }
            }
          }
        }
        // Field s - 2 is complete on this barrier before any warp tells it of field s.
        if (s > 2) ok = ok && tma::mbar_wait_for(&bars[which * 2 + (s & 1)], uint32_t((s - 3) >> 1) & 1u, kJLimitNs);
        if (!__all_sync(0xffffffffu, ok)) return;  // the computing threads' own waits run out
        __syncwarp();  // orders every lane's cells before lane 0's arrival; a vote does not
        if (lane == 0) mbar_arrive(&bars[which * 2 + (s & 1)]);
      }
    };
    // Elements a lane asks for together: as many as it has, up to 16.  1403 x 1177 (10 a
    // lane) takes 0.53 ms in rounds of 8, 0.485 with 16, 0.47 with 12; 1000^2 (8 a lane)
    // 0.394 and 0.425 with 8 and 16.
    if constexpr (sizeof(T) == 4 && CPT == 4) {
      if (columns <= 12 * kStride)
        poll(std::integral_constant<int, 12>{});
      else
        poll(std::integral_constant<int, 16>{});
    } else {
      poll(std::integral_constant<int, sizeof(T) == 8 ? 16 : 8>{});
    }
    return;
  }

  const int seconds = R - H;  // H or H - 1: pairs 0 .. seconds - 1 hold a second row
  const int j0 = 1 + tid * CPT;
  const int c_face = nx - 1 - j0;  // column nx-1 among this thread's columns
  bool act[CPT];
#pragma unroll
  for (int c = 0; c < CPT; ++c) act[c] = j0 + c < nx - 1;
  // What the outer columns of warp w see to the west (0) and east (1), per parity of
  // the field.  Warp 0's west is column 0, a face.
  auto edge = [&](int par, int w, int side) {
    return lay.edge + ((par * (Layout<T, CPT>::kWarps + 2) + w + 1) * 2 + side) * H;
  };
  // Lanes 0 and 31 pass their outer columns on (unless that is column nx-1, which
  // keeps what it held at first).
  const bool gives = lane == 31 || (lane == 0 && c_face != 0);
  const int give_to = lane == 0 ? edge(0, warp - 1, 1) : edge(0, warp + 1, 0);
  const int par_step = edge(1, 0, 0) - edge(0, 0, 0);
  const int takes = edge(0, warp, 0);

  auto cell_of = [&](const T* f, int i, int j) {  // band row i
    const int r = i < R ? i : R;
    return K::cell(k, __ldcg(f + int64_t(r0 + r) * nx + (j < nx ? j : nx - 1)));
  };
  auto pair_of = [&](const T* f, int p, int j) { return K::join(cell_of(f, p, j), cell_of(f, p + H, j)); };
  // The field.  Columns beyond nx-1 and second rows beyond the band hold some value
  // of the array.
  for (int p = 0; p < H; ++p) {
#pragma unroll
    for (int c = 0; c < CPT; ++c) store.put(p * lay.row + c * nt + tid, pair_of(A, p, j0 + c));
    if (lane == 0 || lane == 31) {
      const int j = lane == 0 ? j0 : j0 + CPT - 1;
      store.put(give_to + p, pair_of(A, p, j));
      if (j == nx - 1) store.put(give_to + par_step + p, pair_of(B, p, j));
    }
  }
  __syncthreads();
  for (int q = tid; q < 2 * H; q += nt) {
    const int par = q & 1, p = q >> 1;
    store.put(edge(par, 0, 0) + p, pair_of(par ? B : A, p, 0));
    store.put(p * lay.row + columns + par, pair_of(par ? B : A, p, nx - 1));
  }
  __syncthreads();

  bool ok = true;
  // The halo of field s on a side: field 0's and a wall's are in place, any other
  // arrives behind its barrier.
  auto halo_cell = [&](int which, int s, int c) {
    return K::cell(halo_at(which, s)[K::template halo_index<CPT>(c, tid, nt)]);
  };
  auto accept = [&](int which, int s, Cell (&v)[CPT]) {
    if (s > 0 && !wall(which)) {
      if (ok && !mbar_wait_cluster(&bars[which * 2 + (s & 1)], uint32_t((s - 1) >> 1) & 1u, 2 * kJLimitNs)) {
        atomicOr(&g_jbands_error, 1u);
        ok = false;
      }
      __syncwarp();  // no lane sends, and lets the barrier go on, while another still waits
    }
#pragma unroll
    for (int c = 0; c < CPT; ++c) v[c] = halo_cell(which, s, c);
  };
  const uint32_t halo_next[2] = {in_rank(tma::smem_u32(halo_at(1, 0)), near(0) ? rank - 1 : rank),
                                 in_rank(tma::smem_u32(halo_at(0, 0)), near(1) ? rank + 1 : rank)};
  const uint32_t bars_next[2] = {in_rank(tma::smem_u32(&bars[2]), near(0) ? rank - 1 : rank),
                                 in_rank(tma::smem_u32(&bars[0]), near(1) ? rank + 1 : rank)};
  auto post = [&](int which, int s, const Pair (&v)[CPT], int half) {
    if (wall(which)) return;
    Cell cells[CPT];
#pragma unroll
    for (int c = 0; c < CPT; ++c) cells[c] = K::half(v[c], half);
    if (near(which))
      K::template send<CPT>(halo_next[which] + uint32_t((s & 1) * columns * int(sizeof(typename K::Halo))),
                            bars_next[which] + uint32_t(s & 1) * 8u, tid, nt, cells);
    else
      K::template post<CPT>(box(which, 1 - which, uint32_t(s)), uint32_t(s), tid, nt, cells);
  };
  // Once every thread has taken field s, the barrier waits for field s + 2.
  auto expect_next = [&](int s) {
    if (tid != 0 || s < 1) return;
#pragma unroll
    for (int which = 0; which < 2; ++which)
      if (near(which))
        tma::mbar_arrive_expect_tx(&bars[which * 2 + (s & 1)], columns * sizeof(typename K::Halo));
  };
  // Column c of field s: its slot in pair 0's row (column nx-1 is a face).
  auto slot = [&](int s, int c) { return c == c_face ? columns + (s & 1) : c * nt + tid; };
  // Pair p of field s + 1 from the old pairs at, north and south of it; the warp's
  // outer columns and the band's edges are passed on.
  auto update = [&](int s, int p, const Pair (&cur)[CPT], const Pair (&north)[CPT], const Pair (&south)[CPT]) {
    const int par = s & 1;
    const Pair out_w = store.get(takes + par * par_step + p), out_e = store.get(takes + H + par * par_step + p);
    const Pair west = K::select(lane == 0, out_w, K::up1(cur[CPT - 1]));
    const Pair east = K::select(lane == 31, out_e, K::down1(cur[0]));
    auto w_of = [&](int c) { return c > 0 ? cur[c > 0 ? c - 1 : 0] : west; };
    auto e_of = [&](int c) { return c + 1 < CPT ? cur[c + 1 < CPT ? c + 1 : c] : east; };
    Pair y[CPT];
    typename K::Work open[CPT];
    bool sure = true;
    const bool need_b = p < seconds;
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      y[c] = K::point(k, cur[c], w_of(c), e_of(c), south[c], north[c], open[c]);
      sure = sure && K::sure(open[c], act[c], act[c] && need_b);
    }
    if (!sure)
#pragma unroll
      for (int c = 0; c < CPT; ++c)
        if (!K::sure(open[c], act[c], act[c] && need_b))
          y[c] = K::mend(y[c], open[c], act[c], act[c] && need_b, cur[c], w_of(c), e_of(c), south[c], north[c]);
#pragma unroll
    for (int c = 0; c < CPT; ++c) store.put(p * lay.row + c * nt + tid, y[c]);
    if (gives) store.put(give_to + (1 - par) * par_step + p, K::select(lane == 0, y[0], y[CPT - 1]));
    if (s + 1 < halfsweeps) {
      if (p == 0) post(0, s + 1, y, 0);
      if (p == seconds - 1) post(1, s + 1, y, 1);
      if (p == H - 1 && seconds == 0) post(1, s + 1, y, 0);
    }
  };
  auto dump = [&](T* to) {
    for (int p = 0; p < H; ++p)
#pragma unroll
      for (int c = 0; c < CPT; ++c)
        if (act[c]) {
          const Pair v = store.get(p * lay.row + c * nt + tid);
          to[int64_t(r0 + p) * nx + j0 + c] = K::value(K::half(v, 0));
          if (p < seconds) to[int64_t(r0 + p + H) * nx + j0 + c] = K::value(K::half(v, 1));
        }
  };
  // The halo below lies behind the last second row: in pair `seconds` or, when every
  // pair has a second row, past the last pair.
  auto place_below = [&](int s) {
    Cell below[CPT];
    accept(1, s, below);
    if (seconds < H)
#pragma unroll
      for (int c = 0; c < CPT; ++c) store.put_half(seconds * lay.row + c * nt + tid, 1, below[c]);
  };

  for (int s = 0; s < halfsweeps; s += 2) {
    // Down: the halo above is needed first, the one below last.
    {
      Pair north[CPT], cur[CPT], south[CPT];
      Cell row_h[CPT];  // old row H, south of row H - 1
      int at[CPT];
      accept(0, s, row_h);
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        at[c] = slot(s, c);
        cur[c] = store.get(at[c]);
        north[c] = K::join(row_h[c], K::half(store.get(at[c] + (H - 1) * lay.row), 0));
        row_h[c] = K::half(cur[c], 1);
      }
#pragma unroll 1
      for (int p = 0; p < H; ++p) {
        const bool at_below = p == seconds - 1 || (p == 0 && seconds == 0);
        if (at_below) place_below(s);
#pragma unroll
        for (int c = 0; c < CPT; ++c) at[c] += lay.row;
        if (p + 1 < H) {
#pragma unroll
          for (int c = 0; c < CPT; ++c) south[c] = store.get(at[c]);
        } else {
#pragma unroll
          for (int c = 0; c < CPT; ++c) {
            // Without a second row here that half is not used, and the halo's place may
            // already be the neighbour's again: the last second row has been sent.
            const Cell below = at_below ? halo_cell(1, s, c) : K::half(cur[c], 1);
            south[c] = K::join(seconds == 0 ? below : row_h[c], below);
          }
        }
        update(s, p, cur, north, south);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          north[c] = cur[c];
          cur[c] = south[c];
        }
      }
      if (compute_sync_or(nt, !ok)) return;
      expect_next(s);
    }
    // Up: the halo below first.
    {
      if (s + 2 == halfsweeps) dump(B);
      Pair north[CPT], cur[CPT], south[CPT];
      Cell row_hm1[CPT];  // old row H - 1, north of row H
      int at[CPT];
      place_below(s + 1);
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        at[c] = slot(s + 1, c);
        const Cell below = halo_cell(1, s + 1, c);
        south[c] = K::join(seconds == 0 ? below : K::half(store.get(at[c]), 1), below);
        at[c] += (H - 1) * lay.row;
        cur[c] = store.get(at[c]);
        row_hm1[c] = K::half(cur[c], 0);
      }
#pragma unroll 1
      for (int p = H - 1; p >= 0; --p) {
#pragma unroll
        for (int c = 0; c < CPT; ++c) at[c] -= lay.row;
        if (p > 0) {
#pragma unroll
          for (int c = 0; c < CPT; ++c) north[c] = store.get(at[c]);
        } else {
          Cell above[CPT];
          accept(0, s + 1, above);
#pragma unroll
          for (int c = 0; c < CPT; ++c) north[c] = K::join(above[c], row_hm1[c]);
        }
        update(s + 1, p, cur, north, south);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          south[c] = cur[c];
          cur[c] = north[c];
        }
      }
      if (compute_sync_or(nt, !ok)) return;
      expect_next(s + 1);
    }
  }
  dump(A);
}

// The same half-sweeps in global memory, for a launch without its clusters: rows dealt
// out to `parts` CTAs (all resident, as the launch is cooperative), which meet after
// every half-sweep at `arrived`.
template <typename T>
__device__ __noinline__ void in_memory(T* A, T* B, int ny, int nx, int halfsweeps, int parts, uint32_t* arrived) {
  if (int(blockIdx.x) >= parts) return;
  for (int s = 0; s < halfsweeps; ++s) {
    const T* src = s & 1 ? B : A;
    T* dst = s & 1 ? A : B;
    for (int i = 1 + int(blockIdx.x); i < ny - 1; i += parts)
      for (int j = 1 + int(threadIdx.x); j < nx - 1; j += int(blockDim.x)) {
        const int64_t at = int64_t(i) * nx + j;
        const T* p = src + at;
        T sum = add_rn(__ldcg(p), __ldcg(p - 1));
        sum = add_rn(sum, __ldcg(p + 1));
        sum = add_rn(sum, __ldcg(p + nx));
        sum = add_rn(sum, __ldcg(p - nx));
        __stcg(dst + at, mul_rn(T(0.2), sum));
      }
    __syncthreads();
    if (parts == 1) continue;
    bool ok = true;
    if (threadIdx.x == 0) {
      const uint32_t all = uint32_t(parts) * uint32_t(s + 1);
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrived) : "memory");
      const uint64_t t0 = tma::globaltimer();
      for (;;) {
        uint32_t v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrived) : "memory");
        if (int32_t(v - all) >= 0) break;
        if (tma::globaltimer() - t0 > kJLimitNs) {
          atomicOr(&g_jbands_error, 1u);
          ok = false;
          break;
        }
      }
    }
    if (__syncthreads_or(!ok)) return;
  }
}

// in_cluster: the CTAs of a cluster that base, extra and mail are meant for.
template <typename T, int CPT>
__global__ void __launch_bounds__(kCompute<T, CPT> + 32 * kPollWarps<T>, 1)
jacobi2d_bands(T* __restrict__ A, T* __restrict__ B, int ny, int nx, int halfsweeps, int base, int extra, int nb,
               int in_cluster, typename Kind<T>::Mail* __restrict__ mail, uint32_t* __restrict__ arrived) {
  uint32_t size;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
  if (int(size) != in_cluster) {  // the same for every CTA of the launch
    in_memory<T>(A, B, ny, nx, halfsweeps, int(gridDim.x) > in_cluster ? nb : 1, arrived);
    return;
  }
  if (int(blockIdx.x) < nb)
    run_band<T, CPT>(A, B, ny, nx, halfsweeps, base, extra, nb, mail);
  else
    cluster_sync();
  cluster_sync();  // shared memory stays while a band of the cluster may still send to it
}

// The instances: columns a thread, and the widest grid of each.
template <typename T>
struct Instance {
  using Kernel = void (*)(T*, T*, int, int, int, int, int, int, int, typename Kind<T>::Mail*, uint32_t*);
  Kernel kern;
  int cpt, compute;
  size_t (*bytes)(int H, int threads);
};
template <typename T, int CPT>
constexpr Instance<T> instance() {
  return {jacobi2d_bands<T, CPT>, CPT, kCompute<T, CPT>,
          [](int H, int threads) { return Layout<T, CPT>(H, threads).total; }};
}
template <typename T>
const Instance<T>* instances() {
  if constexpr (sizeof(T) == 8) {
    static const Instance<T> all[3] = {instance<T, 1>(), instance<T, 2>(), instance<T, 3>()};
    return all;
  } else {
    static const Instance<T> all[3] = {instance<T, 2>(), instance<T, 4>(), instance<T, 8>()};
    return all;
  }
}

// Cluster sizes, and how many CTAs of each (one per SM) the device takes at once: on
// 152 SMs 112, 130, 144 and 152, as clusters do not cross GPCs.
constexpr int kClusters[4] = {16, 10, 4, 2};

// Asked of the driver once per device and instance; 0 where it cannot be had.
template <typename T>
int clustered_ctas(int dev, int which, int ci, size_t smem) {
  static std::atomic<int> known[64][3][4];  // 1 + the answer
  std::atomic<int>& slot = known[dev][which][ci];
  if (const int k = slot.load(std::memory_order_acquire)) return k - 1;
  const Instance<T>& in = instances<T>()[which];
  const void* kern = reinterpret_cast<const void*>(in.kern);
  int n = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) == cudaSuccess &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(kClusters[ci]));
    cfg.blockDim = dim3(unsigned(in.compute + 32 * kPollWarps<T>));
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(kClusters[ci]);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) n = 0;
    n *= kClusters[ci];
  }
  if (n == 0) cudaGetLastError();
  slot.store(n + 1, std::memory_order_release);
  return n;
}

}  // namespace

// A pool for the launches that hand values on, kept per device (also jacobi1d_resident.cu).
cudaError_t scratch_pool(cudaMemPool_t* out) {
  static std::mutex mu;
  static cudaMemPool_t pools[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  if (!pools[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t p;
    if ((e = cudaMemPoolCreate(&p, &props)) != cudaSuccess) return e;
    uint64_t keep = uint64_t(64) << 20;  // more than four calls' mail
    cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
    pools[dev] = p;
  }
  *out = pools[dev];
  return cudaSuccess;
}

// Runs the whole time loop of Jacobi-2D in one cooperative launch, or returns
// NPBGB_ERR_STATE, after which the caller uses the chained kernels: when the bands do
// not fit (a band in shared memory, its width in the threads: 1056 columns of
// binary64, 4096 of binary32), on a stream that is being captured (the chained kernels
// need no scratch memory), and, unless asked for every grid that fits
// (NPBGB_CFG_JACOBI_BANDS = 2), where the chained kernels measured faster:
//   * binary64: on values in [0, 1) bands win (300^2, TSTEPS=50: 0.25 against 0.30 ms),
//     but every pair with a value out of the limbs' range is mended out of line, and
//     fields come to hold such values (NPBench's own initial field 0.63 against 0.35, a
//     hot wall in a cold box 0.51 against 0.33, standard normal values 0.64 against 0.39);
//   * binary32 of more than 2049 columns (8 a thread) and fewer rows than 0.29 of them,
//     where a half-sweep gains too little on the load and the way back.  TSTEPS=16 and 40,
//     us, chained and bands: 2300 columns, 600 rows 161, 172 and 380, 367; 750 rows 179,
//     172 and 427, 356; 3300, 750 187, 215 and 442, 454; 900 227, 226 and 553, 479; 4096, 900
//     226, 254 and 544, 546; 1200 265, 273 and 644, 566;
//   * next to a tile queue, whose worker would keep the bands' CTAs waiting;
//   * short runs, as launch, load and way back cost about 25 us and more for wide
//     grids (binary32, TSTEPS=6 and 11: 1000^2 52 and 69 us against 55 and 91; 2500^2
//     164 and 227 against 123 and 229, with 21 358 against 436).
template <typename T>
int32_t jacobi2d_bands_run(T* a, T* b, int64_t ny, int64_t nx, int32_t tsteps, cudaStream_t st) {
  if (g_cfg_jacobi_bands == 0) return NPBGB_ERR_STATE;
  const bool any = g_cfg_jacobi_bands == 2;
  if (tsteps <= 1 || tsteps > (1 << 30) || ny < 4 || nx < 3 || ny > (1 << 20) || nx > 4096) return NPBGB_ERR_STATE;
  if (sizeof(T) == 8 && !(any && g_cfg_f64_emulation)) return NPBGB_ERR_STATE;
  // As few columns a thread as the width allows.
  int which = 0;
  while (which < 3 && nx - 1 > int64_t(instances<T>()[which].cpt) * instances<T>()[which].compute) ++which;
  if (which == 3) return NPBGB_ERR_STATE;
  const Instance<T>& in = instances<T>()[which];
  const bool wide = sizeof(T) == 4 && which == 2;
  if (!any && (tsteps < (!wide ? 8 : nx > 2400 ? 20 : 16) || (wide && 100 * ny < 29 * nx))) return NPBGB_ERR_STATE;
  if (!any && queue_exists()) return NPBGB_ERR_STATE;
  int dev = 0, smem_max = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (dev < 0 || dev >= 64) return NPBGB_ERR_STATE;
  const size_t room = size_t(smem_max) - 1024;
  const int compute = int(cdiv(cdiv(nx - 1, in.cpt), 32) * 32), columns = in.cpt * compute;
  // As few pairs a thread as any cluster size gives, but two (one leaves more bands
  // and their hand-offs: 150^2, binary32, TSTEPS=50 0.147 against 0.136 ms); then the
  // largest clusters.
  const int64_t interior = ny - 2;
  int H = 0, in_cluster = 0;
  for (int ci = 0; ci < 4; ++ci) {
    const int ctas = clustered_ctas<T>(dev, which, ci, room);
    if (ctas < 1) continue;
    const int64_t h = std::max<int64_t>(cdiv(interior, 2 * int64_t(ctas)), 2);
    if (in_cluster == 0 || h < H) H = int(std::min<int64_t>(h, 1 << 20)), in_cluster = kClusters[ci];
  }
  const size_t smem = in_cluster ? in.bytes(H, compute) : 0;
  if (in_cluster == 0 || smem > room) return NPBGB_ERR_STATE;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone)
    return NPBGB_ERR_STATE;
  const int nb = int(cdiv(interior, 2 * H)), clusters = int(cdiv(nb, in_cluster));
  const size_t mail_bytes = size_t(4) * clusters * size_t(columns) * sizeof(typename Kind<T>::Mail);
  const size_t bytes = mail_bytes + 256;  // and a counter
  cudaMemPool_t pool;
  void* scratch = nullptr;
  cudaError_t e;
  if ((e = scratch_pool(&pool)) != cudaSuccess ||
      (e = cudaMallocFromPoolAsync(&scratch, bytes, pool, st)) != cudaSuccess) {
    cudaGetLastError();
    return NPBGB_ERR_STATE;  // no memory for the mail: the chained kernels need none
  }
  if (clusters > 1) e = cudaMemsetAsync(scratch, 0, bytes, st);
  if (e == cudaSuccess) {
    auto* mail = static_cast<typename Kind<T>::Mail*>(scratch);
    auto* arrived = reinterpret_cast<uint32_t*>(static_cast<unsigned char*>(scratch) + mail_bytes);
    int ny_ = int(ny), nx_ = int(nx), hs = 2 * (tsteps - 1), nb_ = nb;
    int base = int(interior / nb), extra = int(interior % nb);
    void* args[] = {&a, &b, &ny_, &nx_, &hs, &base, &extra, &nb_, &in_cluster, &mail, &arrived};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(clusters * in_cluster));
    cfg.blockDim = dim3(unsigned(compute + 32 * kPollWarps<T>));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = unsigned(in_cluster);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    e = launch_together(cfg, reinterpret_cast<const void*>(in.kern), args);
  }
  cudaFreeAsync(scratch, st);
  return e == cudaSuccess ? NPBGB_OK : NPBGB_ERR_STATE;  // not launched
}

template int32_t jacobi2d_bands_run<double>(double*, double*, int64_t, int64_t, int32_t, cudaStream_t);
template int32_t jacobi2d_bands_run<float>(float*, float*, int64_t, int64_t, int32_t, cudaStream_t);

uint32_t take_jacobi_bands_device_error() {
  unsigned int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_jbands_error, sizeof(v)) != cudaSuccess) return 0xffffffffu;
  if (v) cudaMemcpyToSymbol(g_jbands_error, &zero, sizeof(zero));
  return v;
}

}  // namespace npbgb
