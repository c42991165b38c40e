// prx_device.cuh -- device helpers shared by the kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "prx_internal.h"
#include "prx_softadd.h"

namespace prx {

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// Row segments (see GraphDev): index of row v's begin in the offsets, and
// the start of its segment's edges.  shift 32 / base null: the plain CSR.
__device__ __forceinline__ uint64_t seg_index(uint32_t v, uint32_t shift) {
  return (uint64_t)v + ((uint64_t)v >> shift);
}
__device__ __forceinline__ const uint32_t* seg_edges(const uint32_t* edg, const unsigned long long* base, uint32_t shift,
                                                     uint32_t v) {
  return base ? edg + base[(uint64_t)v >> shift] : edg;
}
__device__ __forceinline__ uint32_t row_len(const uint32_t* __restrict__ off, uint32_t shift, uint32_t v) {
  const uint64_t i = seg_index(v, shift);
  return off[i + 1] - off[i];
}

// In-degree class of v (see kLowMax).
__device__ __forceinline__ int in_class(const uint32_t* __restrict__ xtoff, uint32_t shift, uint32_t v,
                                        uint32_t mid_max) {
  const uint32_t d = row_len(xtoff, shift, v);
  return d <= kLowMax ? LOW : (d <= mid_max ? MID : HIGH);
}

// Set bit v of a bitmap; true if this call changed it from 0 to 1.  Bits only
// go 0 -> 1 while marking kernels run, so a set bit seen by the plain load is
// final and the atomic can be skipped.
__device__ __forceinline__ bool test_and_set(uint32_t* bm, uint32_t v) {
  const uint32_t bit = 1u << (v & 31u);
  if (bm[v >> 5] & bit) return false;
  return !(atomicOr(&bm[v >> 5], bit) & bit);
}

__device__ __forceinline__ void clear_bit(uint32_t* bm, uint32_t v) {
  atomicAnd(&bm[v >> 5], ~(1u << (v & 31u)));
}

// Append v to list/cnt.  Lanes of the active set that append to the same
// counter share one atomicAdd (safe under divergence).
__device__ __forceinline__ void push(uint32_t* list, uint32_t* cnt, uint32_t v) {
  const unsigned active = __activemask();
  const unsigned peers = __match_any_sync(active, (unsigned long long)(uintptr_t)cnt);
  const int leader = __ffs(peers) - 1;
  const unsigned lane = lane_id();
  uint32_t base = 0;
  if ((int)lane == leader) base = atomicAdd(cnt, (uint32_t)__popc(peers));
  base = __shfl_sync(peers, base, leader);
  list[base + __popc(peers & ((1u << lane) - 1u))] = v;
}

// *cnt += 1 by every active lane, one atomic for them together.
__device__ __forceinline__ void count_one(uint32_t* cnt) {
  const unsigned active = __activemask();
  if ((int)lane_id() == __ffs(active) - 1) atomicAdd(cnt, (uint32_t)__popc(active));
}

// Block-wide max of a non-negative double given as its bit pattern (for
// x >= 0 the IEEE-754 bit patterns order like the values), folded into *dst
// with one atomicMax per block.  Every thread of the block must call it; the
// leading barrier lets calls follow one another (warp 0 may still be reading
// the shared slots of the previous call).
__device__ __forceinline__ void block_max_bits(unsigned long long x, unsigned long long* dst) {
  __shared__ unsigned long long smax[32];
  for (int o = 16; o; o >>= 1) {
    const unsigned long long y = __shfl_xor_sync(0xffffffffu, x, o);
    x = y > x ? y : x;
  }
  const int w = threadIdx.x >> 5;
  __syncthreads();
  if (lane_id() == 0) smax[w] = x;
  __syncthreads();
  if (w == 0) {
    x = lane_id() < (blockDim.x >> 5) ? smax[lane_id()] : 0ull;
    for (int o = 16; o; o >>= 1) {
      const unsigned long long y = __shfl_xor_sync(0xffffffffu, x, o);
      x = y > x ? y : x;
    }
    if (lane_id() == 0 && x) atomicMax(dst, x);
  }
}

// The same for a non-negative float given as its bit pattern.
__device__ __forceinline__ void block_max_u32(unsigned int x, unsigned int* dst) {
  __shared__ unsigned int smax[32];
  for (int o = 16; o; o >>= 1) x = max(x, __shfl_xor_sync(0xffffffffu, x, o));
  const int w = threadIdx.x >> 5;
  __syncthreads();
  if (lane_id() == 0) smax[w] = x;
  __syncthreads();
  if (w == 0) {
    x = lane_id() < (blockDim.x >> 5) ? smax[lane_id()] : 0u;
    for (int o = 16; o; o >>= 1) x = max(x, __shfl_xor_sync(0xffffffffu, x, o));
    if (lane_id() == 0 && x) atomicMax(dst, x);
  }
}

__device__ __forceinline__ void block_sum_u64(unsigned long long x, unsigned long long* dst) {
  __shared__ unsigned long long ssum[32];
  for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  const int w = threadIdx.x >> 5;
  __syncthreads();
  if (lane_id() == 0) ssum[w] = x;
  __syncthreads();
  if (w == 0) {
    x = lane_id() < (blockDim.x >> 5) ? ssum[lane_id()] : 0ull;
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane_id() == 0 && x) atomicAdd(dst, x);
  }
}

__device__ __forceinline__ void block_sum_u32(uint32_t x, uint32_t* dst) {
  __shared__ uint32_t ssum[32];
  x = __reduce_add_sync(0xffffffffu, x);
  __syncthreads();
  if (lane_id() == 0) ssum[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x < 32) {
    x = __reduce_add_sync(0xffffffffu, lane_id() < (blockDim.x >> 5) ? ssum[lane_id()] : 0u);
    if (lane_id() == 0 && x) atomicAdd(dst, x);
  }
}

// Barrier over all blocks of a cooperative launch (st->bar zero before it).
// Thread 0 counts the block in and polls; every write of the block before the
// barrier is visible to every block after it (thread 0's release and acquire
// order the blocks, the block barriers the other threads).  The wait is
// bounded: after kGridSpin polls (seconds; a phase takes well under a
// millisecond), or when another block gave up, sync returns false in every
// thread and the kernel must return.  after(): run by thread 0 once all
// blocks have arrived, before the block continues.
constexpr int kGridSpin = 1 << 23;
struct GridBarrier {
  State* st;
  uint32_t target = 0;
  __device__ explicit GridBarrier(State* s) : st(s) {}
  template <class F>
  __device__ bool sync(F after) {
    __shared__ int ok;
    target += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&st->bar) : "memory");
      auto arrived = [&] {
        uint32_t n;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(&st->bar) : "memory");
        return n;
      };
      int good = 1;
      for (int spin = 0; (int)(arrived() - target) < 0;) {
        if (++spin > kGridSpin || ((spin & 1023) == 0 && (*(volatile uint32_t*)&st->err & kErrGridWait))) {
          atomicOr(&st->err, kErrGridWait);
          good = 0;
          break;
        }
      }
      if (good) after();
      ok = good;
    }
    __syncthreads();
    return ok != 0;
  }
};

// The units (MID rows, words of LOW rows) of a cooperative loop are shared out
// over its warps from the last one backwards, nlong long rows over its blocks from
// the first on, so that the blocks that hold them get the last units.  Very long
// rows (solo) go the other way round: a cooperative launch fills four SMs with its
// first blocks, three each, and the last blocks are on SMs of their own; and where
// they are a few of the grid's, their blocks take no units: 20 rows of 500,000 among
// a million vertices, Static 7.1 | 2.8 ms, DF-P 23.6 | 8.4.
struct WarpShare {
  uint32_t all, any;     // warps of the grid, and this one among them
  uint32_t warps, warp;  // those that take units, and this one among them (at least 2^31: it takes none)
  uint32_t row;          // this block's first long row
  __device__ __forceinline__ WarpShare(uint32_t nlong, bool solo) {
    const uint32_t per = blockDim.x >> 5, back = gridDim.x - 1 - blockIdx.x;
    const uint32_t lb = solo && 4ull * nlong <= gridDim.x ? nlong : 0u;
    row = solo ? back : blockIdx.x;
    all = gridDim.x * per;
    any = (solo ? blockIdx.x : back) * per + (threadIdx.x >> 5);
    warps = (gridDim.x - lb) * per;
    warp = any < warps ? any : 0x80000000u;
  }
};

__device__ __forceinline__ unsigned long long dbits(double x) {
  return (unsigned long long)__double_as_longlong(x);
}

// GB300 executes two FP64 lanes per SM per clock, so one warp-wide FP64
// instruction costs as much pipe time as dozens of integer ones: the helpers
// below keep to the FP64 operations the reference's arithmetic needs and do
// conversions and comparisons on bit patterns.

// (double)d exactly, from integer operations: d = 2^e * 1.f with e the
// position of the leading one.
__device__ __forceinline__ double u32_to_f64(uint32_t d) {
  const uint32_t lz = __clz(d);  // 32 for d == 0
  const unsigned long long frac = ((unsigned long long)d << (21 + (lz & 31))) & ((1ull << 52) - 1);
  const unsigned long long bits = ((unsigned long long)(1054 - lz) << 52) | frac;  // 1023 + (31 - lz)
  return d ? __longlong_as_double((long long)bits) : 0.0;
}

// a / d correctly rounded, for an integer d >= 1 and y = RN(1/d), by
// Markstein's method (P. Markstein, "IA-64 and Elementary Functions", 2000):
// q = RN(a*y) is within one ulp of a/d, so r = a - q*d is exact in one fma,
// and RN(q + r*y) is the correctly rounded quotient.  Three FP64 operations
// instead of a full division; valid while nothing over- or underflows (ranks
// and contributions here are far from both).  Checked bit for bit against
// the IEEE division by prx_selftest.
__device__ __forceinline__ double div_count(double a, uint32_t d, double y) {
  const double q = a * y;
  const double r = fma(-q, u32_to_f64(d), a);
  return fma(r, y, q);
}

// The relative-change tests of the frontier modes, RN(x / m) <= c and
// RN(x / m) > c with x = |a - b| and m = fmax(a, b).  For non-negative finite
// a, b (the ranks) m is the larger bit pattern, and non-negative doubles
// order as their bit patterns: away from a band of 64 ulps around RN(c*m)
// the exact quotient is more than an ulp of c from c (the product's rounding
// is one half ulp), so its rounding lies on the same side, and one FP64
// multiplication decides.  Inside the band, or for negative, infinite or NaN
// operands or a subnormal c*m, the quotient is formed as written.
struct RelChange {
  double x, m;
  bool fast;
};
__device__ __forceinline__ RelChange rel_change(double a, double b) {
  const long long ab = __double_as_longlong(a), bb = __double_as_longlong(b);
  RelChange r;
  r.x = fabs(a - b);
  r.fast = (ab | bb) >= 0 && __double_as_longlong(r.x) < 0x7ff0000000000000ll;
  r.m = r.fast ? __longlong_as_double(ab > bb ? ab : bb) : fmax(a, b);
  return r;
}
constexpr long long kRelBand = 64;
__device__ __forceinline__ int rel_side(const RelChange& r, double c) {  // -1 below c, +1 above, 0 undecided
  if (!r.fast) return 0;
  const long long xb = __double_as_longlong(r.x), cb = __double_as_longlong(c * r.m);
  if (cb < (1ll << 52)) return 0;  // c*m subnormal or zero
  return xb < cb - kRelBand ? -1 : (xb > cb + kRelBand ? 1 : 0);
}
__device__ __forceinline__ bool quot_le(const RelChange& r, double c) {
  const int side = rel_side(r, c);
  return side ? side < 0 : r.x / r.m <= c;
}
__device__ __forceinline__ bool quot_gt(const RelChange& r, double c) {
  const int side = rel_side(r, c);
  return side ? side > 0 : r.x / r.m > c;
}

// FP32 rounds of the refinement stop once the change they predict for their
// next sweep -- this sweep's change times the larger of its last two ratios
// to the sweep before (the observed rate of the Jacobi iteration) -- is below
// kPredictSafety times the tolerance: the FP64 residual sweep that follows
// measures about that next change, so it passes without the FP32 sweep that
// would only confirm it.  The FP64 test still decides convergence; a wrong
// prediction costs one more round, never accuracy.  prev / prev2: the
// changes of the two sweeps before (0: none yet).
constexpr float kPredictSafety = 0.8f;
__device__ __forceinline__ bool fp32_round_done(float change, float prev, float prev2, double tol) {
  if (!(prev > 0.f && prev2 > 0.f && change < prev && prev < prev2)) return false;
  const float rate = fmaxf(change / prev, prev / prev2);
  return change * rate < kPredictSafety * (float)tol;
}

// Edge id as stored in a layout: a hot source's number with the flag, else
// the id itself (hot_idx null: plain ids; see GraphDev::hot_idx, of a graph
// of `words` bitmap words).
__device__ __forceinline__ uint32_t layout_id(const uint32_t* __restrict__ hot_idx, uint32_t words, uint32_t u) {
  if (!hot_idx) return u;
  const uint32_t w = __ldg(hot_idx + (u >> 5)), below = w & ((1u << (u & 31u)) - 1u);
  return ((w >> (u & 31u)) & 1u) ? (kHotFlag | (__ldg(hot_idx + words + (u >> 5)) + __popc(below))) : u;
}

// The contribution of edge id u: with `hot` (a layout whose hot sources are
// encoded, kHotFlag | number) from the dense hot copy ch, else c[u].
// COH: c is written by other blocks of the same launch (between grid
// barriers), so the load is an ordinary one, not the read-only path.
template <class T, bool COH = false>
__device__ __forceinline__ T gather(const T* c, const T* ch, bool hot, uint32_t u) {
  const T* at = (hot && (u & kHotFlag)) ? ch + (u ^ kHotFlag) : c + u;
  if constexpr (COH) return *at;
  else return __ldg(at);
}

// Sum of c[edg[j]] for j in [s, e) added front to back onto acc.  The edge
// ids are read as aligned 16-byte groups of four (edg must be 16-byte
// aligned and allocated per edge_slots); ids outside [s, e) in the first and
// last group are loaded but neither gathered nor added.  Four gathers are in
// flight per group.  hot / ch: see gather().
template <class T>
__device__ __forceinline__ T lane_row_sum(const T* __restrict__ c, const uint32_t* __restrict__ edg, uint32_t s,
                                          uint32_t e, T acc, const T* __restrict__ ch = nullptr, bool hot = false) {
  if (s >= e) return acc;
  uint32_t j = s & ~3u;
  if (j < s) {  // head group: ids j+1 .. j+3 from s on
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(edg + j));
    const bool b1 = s <= j + 1 && j + 1 < e, b2 = s <= j + 2 && j + 2 < e, b3 = j + 3 < e;
    const T c1 = b1 ? gather(c, ch, hot, u.y) : T(0), c2 = b2 ? gather(c, ch, hot, u.z) : T(0),
            c3 = b3 ? gather(c, ch, hot, u.w) : T(0);
    if (b1) acc += c1;
    if (b2) acc += c2;
    if (b3) acc += c3;
    j += 4;
  }
  for (; j + 4 <= e; j += 4) {
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(edg + j));
    const T c0 = gather(c, ch, hot, u.x), c1 = gather(c, ch, hot, u.y), c2 = gather(c, ch, hot, u.z),
            c3 = gather(c, ch, hot, u.w);
    acc += c0; acc += c1; acc += c2; acc += c3;
  }
  if (j < e) {  // tail group: ids j .. e-1 (at most 3)
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(edg + j));
    const bool b1 = j + 1 < e, b2 = j + 2 < e;
    const T c0 = gather(c, ch, hot, u.x), c1 = b1 ? gather(c, ch, hot, u.y) : T(0),
            c2 = b2 ? gather(c, ch, hot, u.z) : T(0);
    acc += c0;
    if (b1) acc += c1;
    if (b2) acc += c2;
  }
  return acc;
}

// a / d correctly rounded for an integer d >= 1: in integer operations
// (quot_bits) with R = the table's reciprocal (0: no entry), otherwise -- a
// not a positive normal of the middle range, or the estimate undecided -- by
// div_count with y = RN(1/d) loaded from *y.
__device__ __forceinline__ double div_outdeg(double a, uint32_t d, uint64_t R, const double* y) {
  bool undecided;
  const uint64_t q = quot_bits((uint64_t)__double_as_longlong(a), d, R, &undecided);
  if (undecided || R == 0 || (uint32_t)__double2hiint(a) - kQuotMinHi >= kQuotHiRange) return div_count(a, d, *y);
  return __longlong_as_double((long long)q);
}

// Whether soft_add takes every lane's sum and terms (one vote).
__device__ __forceinline__ bool soft_step(double acc, const double x[4]) {
  const uint32_t h0 = (uint32_t)__double2hiint(x[0]), h1 = (uint32_t)__double2hiint(x[1]),
                 h2 = (uint32_t)__double2hiint(x[2]), h3 = (uint32_t)__double2hiint(x[3]);
  const uint32_t top = max(max(h0, h1), max(h2, h3)), ha = (uint32_t)__double2hiint(acc);
  return __all_sync(0xffffffffu, ha - kSoftMinHi < kSoftAddHiLimit - kSoftMinHi && top < kSoftAddHiLimit);
}

// The adds of a step, x[LO .. m) in order (m, at most 4, the same in every
// lane), the first K of them by soft_add where it takes them, the others
// DADDs.  The bits are the same.
template <int K, int LO>
__device__ __forceinline__ double add_step(double acc, const double x[4], uint32_t m) {
  if (K > 0 && soft_step(acc, x)) {
    SoftAcc u = soft_unpack((uint64_t)__double_as_longlong(acc));
#pragma unroll
    for (int i = LO; i < LO + K && i < 4; ++i)
      if (m > (uint32_t)i) u = soft_add(u, (uint64_t)__double_as_longlong(x[i]));
    acc = __longlong_as_double((long long)soft_pack(u));
#pragma unroll
    for (int i = LO + K; i < 4; ++i)
      if (m > (uint32_t)i) acc += x[i];
  } else {
#pragma unroll
    for (int i = LO; i < 4; ++i)
      if (m > (uint32_t)i) acc += x[i];
  }
  return acc;
}

// FP64 row sums, one row per lane, for a whole warp: every lane calls it
// (lanes with nothing to add pass s == e).  Each lane adds c[edg[j]] for j in
// [s, e) onto init front to back, as lane_row_sum does, but the warp issues
// exactly L adds, L the longest row: lane_row_sum's aligned head and tail
// groups take up to three predicated adds each, and predicated-off FP64
// instructions cost the warp as much as live ones.  Step k reads ids
// s+4k .. s+4k+3 out of the two aligned 16-byte groups they span (the lane's
// offset s & 3 picks them), loaded a step ahead; a lane past its row's end
// adds +0.0, which leaves the sum (of non-negative terms from +0) unchanged.
// ZERO: init is +0, so the first term is the first sum and is not added.
// K of every step's four adds are soft_adds, so that the FP64 pipe carries
// fewer of them.
// AHEAD: steps whose gathers are in flight beyond the one being added, for
// launches with few warps a scheduler, where a step's latency (ids, gathers
// and four dependent adds) is what counts; 8 registers each.
template <bool COH, bool ZERO, int AHEAD, int K>
__device__ __forceinline__ double warp_row_sums(const double* c, const uint32_t* __restrict__ edg, uint32_t s,
                                                uint32_t e, double init, const double* ch, bool hot) {
  const uint32_t len = e - s;
  const uint32_t L = __reduce_max_sync(0xffffffffu, len);
  if (L == 0) return init;
  const uint32_t j0 = s & ~3u, o = s & 3u;
  auto ids = [&](uint32_t t) {  // the group at step t of this lane's row
    const uint32_t j = j0 + t;
    return len && j < e ? __ldg(reinterpret_cast<const uint4*>(edg + j)) : make_uint4(0, 0, 0, 0);
  };
  auto terms = [&](uint32_t t, const uint4& g0, const uint4& g1, double x[4]) {
    // ids at s+t+i, i < 4: the 8 words of g0:g1 shifted by o
    const bool o1 = o & 1u, o2 = o & 2u;
    const uint32_t a0 = o1 ? g0.y : g0.x, a1 = o1 ? g0.z : g0.y, a2 = o1 ? g0.w : g0.z, a3 = o1 ? g1.x : g0.w,
                   a4 = o1 ? g1.y : g1.x, a5 = o1 ? g1.z : g1.y;
    const uint32_t u0 = o2 ? a2 : a0, u1 = o2 ? a3 : a1, u2 = o2 ? a4 : a2, u3 = o2 ? a5 : a3;
    x[0] = t < len ? gather<double, COH>(c, ch, hot, u0) : 0.0;
    x[1] = t + 1 < len ? gather<double, COH>(c, ch, hot, u1) : 0.0;
    x[2] = t + 2 < len ? gather<double, COH>(c, ch, hot, u2) : 0.0;
    x[3] = t + 3 < len ? gather<double, COH>(c, ch, hot, u3) : 0.0;
  };
  // lanes without terms sum from 1 (in soft_add's range) and return init
  double acc = len ? init : 1.0;
  auto first = [&](const double x[4]) {  // step 0
    const uint32_t m = min(4u, L);
    if (!ZERO) return add_step<K, 0>(acc, x, m);
    const double x0 = __double_as_longlong(x[0]) == (long long)(1ull << 63) ? 0.0 : x[0];  // +0 + -0 = +0
    return add_step<K, 1>(len ? x0 : 1.0, x, m);
  };
  uint4 g0 = ids(0), g1 = ids(4);
  if constexpr (AHEAD > 0) {
    uint4 g2 = ids(8);
    double x[AHEAD + 1][4];  // x[i]: the terms of step t / 4 + i
    auto next = [&](uint32_t t, double y[4]) {  // the terms at t; g0 : g1 hold its ids, g2 the group after
      terms(t, g0, g1, y);
      g0 = g1;
      g1 = g2;
      g2 = ids(t + 12);
    };
#pragma unroll
    for (int i = 0; i <= AHEAD; ++i) next(4 * i, x[i]);
    acc = first(x[0]);
    uint32_t t = 4;
    for (; t + 4 <= L; t += 4) {
#pragma unroll
      for (int k = 0; k < AHEAD; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) x[k][i] = x[k + 1][i];
      next(t + 4 * AHEAD, x[AHEAD]);
      acc = add_step<K, 0>(acc, x[0], 4);
    }
    if (t < L) acc = add_step<K, 0>(acc, x[1], L - t);
  } else {
    double x[4];
    terms(0, g0, g1, x);
    uint4 g2 = ids(8);
    acc = first(x);
    uint32_t t = 4;
    for (; t + 4 <= L; t += 4) {
      g0 = g1;
      g1 = g2;
      terms(t, g0, g1, x);
      g2 = ids(t + 8);
      acc = add_step<K, 0>(acc, x, 4);
    }
    if (t < L) {
      terms(t, g1, g2, x);
      acc = add_step<K, 0>(acc, x, L - t);
    }
  }
  return len ? acc : init;
}

// The same sums of a word's rows laid out as WordRows (from group `base` on):
// len the lane's row, mine whether it is summed.
template <int K>
__device__ __forceinline__ double word_row_sums(const double* c, const uint4* __restrict__ grp, uint32_t base,
                                                uint32_t len, bool mine, const double* ch, bool hot) {
  const uint32_t want = mine ? len : 0u;
  const uint32_t L = __reduce_max_sync(0xffffffffu, want);
  if (L == 0) return 0.0;
  const uint32_t below = (1u << lane_id()) - 1u;
  auto ids = [&](uint32_t t) {  // step t's group, called for 0, 4, 8, ...
    const unsigned rows = __ballot_sync(0xffffffffu, t < len);
    const uint4 u = t < want ? __ldg(grp + (base + __popc(rows & below))) : make_uint4(0, 0, 0, 0);
    base += __popc(rows);
    return u;
  };
  auto terms = [&](uint32_t t, const uint4& u, double x[4]) {
    x[0] = t < want ? gather<double>(c, ch, hot, u.x) : 0.0;
    x[1] = t + 1 < want ? gather<double>(c, ch, hot, u.y) : 0.0;
    x[2] = t + 2 < want ? gather<double>(c, ch, hot, u.z) : 0.0;
    x[3] = t + 3 < want ? gather<double>(c, ch, hot, u.w) : 0.0;
  };
  double x[4];
  uint4 g1 = ids(0), g2 = ids(4);
  terms(0, g1, x);
  g1 = g2;
  g2 = ids(8);
  const double x0 = __double_as_longlong(x[0]) == (long long)(1ull << 63) ? 0.0 : x[0];  // +0 + -0 = +0
  double acc = add_step<K, 1>(want ? x0 : 1.0, x, min(4u, L));  // lanes without terms: in soft_add's range
  uint32_t t = 4;
  for (; t + 4 <= L; t += 4) {
    terms(t, g1, x);
    g1 = g2;
    g2 = ids(t + 8);
    acc = add_step<K, 0>(acc, x, 4);
  }
  if (t < L) {
    terms(t, g1, x);
    acc = add_step<K, 0>(acc, x, L - t);
  }
  return want ? acc : 0.0;
}

}  // namespace prx
