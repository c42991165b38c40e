// prx_update.cuh -- the rank update of one vertex and the row sums of the
// MID and HIGH classes, shared by the launched sweeps (prx_update.cu) and the
// persistent loop (prx_persist.cu).
#pragma once
#include <type_traits>
#include "prx_device.cuh"

namespace prx {

template <int MODE> struct ModeTraits {
  static constexpr bool F32 = (MODE & MODE_F32) != 0;
  static constexpr int BASE = MODE & ~MODE_F32;
  static constexpr bool REFINE = BASE == MODE_REFINE64;
  static constexpr bool DYN = !REFINE && BASE >= PRX_DYNAMIC_TRAVERSAL;
  static constexpr bool FRONTIER = DYN && BASE >= PRX_DYNAMIC_FRONTIER;
  static constexpr bool PRUNE = BASE == PRX_PRUNE_DYNAMIC_FRONTIER;
  using V = typename std::conditional<F32, float, double>::type;  // rank / contribution type
  // resident blocks of 256 per SM the LOW kernel is compiled (40 registers a
  // thread) and launched for.  Static, us a sweep at 7 | 6 | 5: web-like 20M
  // 2591 | 2310 | 2297, 3M 351 | 323 | 318, grid 4096^2 342 | 342 | 380.
  static constexpr int LOW_BLOCKS = 6;
};

// Rank, contribution and carried-sum arrays of a mode: FP64 r / c / acc64,
// or for the FP32 dynamic phase e / ce / acc32.
template <int MODE>
__device__ __forceinline__ typename ModeTraits<MODE>::V* ranks_of(const SolveArgs& a, int p) {
  if constexpr (ModeTraits<MODE>::F32) return a.e[p];
  else return a.r[p];
}
template <int MODE>
__device__ __forceinline__ typename ModeTraits<MODE>::V* contribs_of(const SolveArgs& a, int p) {
  if constexpr (ModeTraits<MODE>::F32) return a.ce[p];
  else return a.c[p];
}
template <int MODE>
__device__ __forceinline__ typename ModeTraits<MODE>::V* carried_of(const SolveArgs& a) {
  if constexpr (ModeTraits<MODE>::F32) return a.acc32;
  else return a.acc64;
}

// Data parity read by an iteration: the refinement's FP64 sweep always reads
// the base ranks (parity 0) and writes parity 1.
template <int MODE>
__device__ __forceinline__ int data_parity(const State* st) {
  return ModeTraits<MODE>::REFINE ? 0 : (st->iter & 1);
}

__device__ __forceinline__ void set_bit(uint32_t* bm, uint32_t w) {
  const uint32_t bit = 1u << (w & 31u);
  if (!(bm[w >> 5] & bit)) atomicOr(&bm[w >> 5], bit);
}

// What an FP64 update of a vertex reads besides its row (loaded before the
// row where latency counts).
struct VertexIn {
  uint32_t d;      // out-degree
  uint64_t R;      // its reciprocal from the table (0: none)
  double r;        // rank before the update
};
__device__ __forceinline__ VertexIn load_vertex(const SolveArgs& a, uint32_t v, int p) {
  VertexIn x;
  x.d = __ldg(a.xtdat + v);
  x.r = a.r[p][v];
  x.R = x.d < kQuotTable ? __ldg(a.qtab + x.d) : 0ull;
  return x;
}

// Finish vertex v given its contribution sum.  Returns |a_v - r_v| as bits
// (of a double; an FP32 change converts exactly).  survive (dynamic): v stays
// affected next iteration; changed (DF / DF-P): its relative change exceeded
// the frontier tolerance, so its out-neighbours become affected (:106-107,
// expanded after the sweep as at :686-687).  FP32 phase: *mag is raised to
// |a_v| (bits of a float).
template <int MODE>
__device__ __forceinline__ unsigned long long finish_vertex(const SolveArgs& a, uint32_t v,
                                                            typename ModeTraits<MODE>::V cv, int p, bool& survive,
                                                            bool& changed, unsigned int& mag, const VertexIn& in) {
  using T = ModeTraits<MODE>;
  if constexpr (T::F32) {
    const uint32_t d = a.xtdat[v];
    const float P = (float)a.P, C0 = (float)a.C0, df = (float)d;
    const float rv = a.e[p][v];
    float av;
    // ce[p][v] is rv / df, formed when rv was (the same division)
    if (T::PRUNE) av = fmaf(P, cv - a.ce[p][v], C0) * (1.f / (1.f - P / df));
    else          av = fmaf(P, cv, C0);
    const float ev = fabsf(av - rv);
    a.e[p ^ 1][v] = av;
    a.ce[p ^ 1][v] = av / df;
    mag = max(mag, __float_as_uint(fabsf(av)));
    survive = true;
    changed = false;
    if (T::FRONTIER) {  // relative change against the tolerances, without the division
      const float m = fmaxf(rv, av);
      if (T::PRUNE && ev <= (float)a.C * m) survive = false;
      changed = ev > (float)a.D * m;
    }
    return dbits((double)ev);
  } else {
    const uint32_t d = in.d;
    const double rv = in.r;
    double av;
    // c[p][v] is RN(rv / d), formed when rv was; pf: 1 / (1 - P/d)
    if (T::PRUNE) av = fma(a.P, cv - a.c[p][v], a.C0) * a.pf[v];
    else          av = fma(a.P, cv, a.C0);
    const double ev = fabs(av - rv);
    a.r[p ^ 1][v] = av;
    if (T::REFINE) {
      // residual of the base ranks, the first FP32 correction and its contribution
      const float rho = (float)(av - rv);
      a.rho[v] = rho;
      a.e[0][v] = rho;
      a.ce[0][v] = __fdividef(rho, (float)d);
    } else {
      a.c[p ^ 1][v] = div_outdeg(av, d, in.R, a.rcp + v);
    }
    survive = true;
    changed = false;
    if constexpr (T::FRONTIER) {  // rel = ev / max(rv, av) compared with C and D
      const RelChange rc = rel_change(av, rv);
      if (T::PRUNE && quot_le(rc, a.C)) survive = false;  // :106
      changed = quot_gt(rc, a.D);                          // :107
    }
    return dbits(ev);
  }
}

// DF keeps every vertex it ever marked affected (only DF-P prunes), so a
// vertex whose out-neighbours were marked once -- as a seed of the batch or by
// an earlier iteration's expansion -- need not be expanded again: the bitmap
// naff, which the marking leaves with its seeds, collects them, and only the
// vertices new to it are.  DF on R-MAT 2^18 in the persistent loop (50
// iterations, nearly every vertex changing in most of them): 5.5 -> 3.0 ms.
// chg: the changed
// vertices of word w (the same in every lane); returns those to expand.
template <bool PRUNE>
__device__ __forceinline__ unsigned fresh_changes(uint32_t* naff, uint32_t w, unsigned chg, uint32_t lane) {
  if (PRUNE || !chg) return chg;
  const unsigned fresh = chg & ~naff[w];
  __syncwarp();
  if (lane == 0 && fresh) atomicOr(&naff[w], fresh);
  return fresh;
}

// Whether to expand nf changed vertices by pulling, when `marked` of the n
// vertices are affected.  A push reads every out-edge of the nf vertices, a
// pull the in-edges of the unmarked ones up to the first changed source: pull
// when more than 1/16 of the vertices changed (pull_threshold) or when more
// changed than are unmarked.  Without the second rule DF on a web-like graph
// of 1.5M vertices, most of them marked from the start, took 1.57 ms of
// launched iterations; with it 1.33 ms.
__device__ __forceinline__ bool expand_by_pull(uint32_t nf, uint32_t marked, uint32_t n, uint32_t pull_threshold) {
  if (pull_threshold == 0xffffffffu) return false;
  return nf > pull_threshold || nf > n - marked;
}

// A contribution: through the read-only path, or with COH (the array is
// written by other blocks of the same launch, between grid barriers) by an
// ordinary load.
template <bool COH, class V>
__device__ __forceinline__ V load_c(const V* c) {
  if constexpr (COH) return *c;
  else return __ldg(c);
}

// The integer pipes take about half of the FP64 adds of the MID sums
// (soft_add): GB300's FP64 pipe needs 20 cycles a warp-wide add, soft_add 14
// of the integer pipes'.  It needs every term to be normal and below 2^977;
// sums that meet another one (zero, negative, subnormal, huge: a caller's
// ranks) are formed again by FP64 adds.  A slot without a term holds +0.0,
// whose unpacked form vanishes against any term; two empty slots give 2^-1022
// and more, which vanishes too, and the sum asked for has at least one term.
__device__ __forceinline__ double soft_plus(double a, double b) {
  return __longlong_as_double((long long)soft_pack(
      soft_add(soft_unpack((uint64_t)__double_as_longlong(a)), (uint64_t)__double_as_longlong(b))));
}
__device__ __forceinline__ bool soft_out_of_range(double x) {
  return (uint32_t)__double2hiint(x) - kSoftMinHi >= kSoftAddHiLimit - kSoftMinHi;
}

// a + b by the FP64 pipe or, with SOFT, the integer pipes.
template <bool SOFT, class V>
__device__ __forceinline__ V plus(V a, V b) {
  if constexpr (SOFT) return soft_plus(a, b);
  else return a + b;
}

// The 32 lane values of up to four rows folded together: x[l] + x[l ^ 16], then
// 8, 4, 2, 1, as a warp's shuffles would fold one row.  Lane 8r + i adds up
// row r's values i, i + 8, i + 16, i + 24 by itself, so four rows take six
// warp-wide FP64 adds instead of twenty (and their epilogues run side by
// side).  One tree per warp; its rows lie 40 doubles apart (no bank conflicts).
struct RowTree {
  static constexpr uint32_t kRows = 4, kStride = 40, kSlots = kRows * kStride;
  double* s;
  __device__ __forceinline__ void put(uint32_t row, double x) const { s[row * kStride + lane_id()] = x; }
  // Row r's sum in lane 8r (r < rows); every lane calls it.
  template <bool SOFT>
  __device__ __forceinline__ double fold(uint32_t rows) const {
    __syncwarp();
    const uint32_t row = lane_id() >> 3;
    const double* x = s + row * kStride + (lane_id() & 7u);
    const bool in = row < rows;
    const double x0 = in ? x[0] : 0.0, x1 = in ? x[8] : 0.0, x2 = in ? x[16] : 0.0, x3 = in ? x[24] : 0.0;
    __syncwarp();
    double z = (x0 + x2) + plus<SOFT>(x1, x3);
    z = plus<SOFT>(z, __shfl_xor_sync(0xffffffffu, z, 4));
    z += __shfl_xor_sync(0xffffffffu, z, 2);
    return plus<SOFT>(z, __shfl_xor_sync(0xffffffffu, z, 1));
  }
};

// MID: the reference's 256-way sum of c over the d ids at ed, by one warp.
// Lane l owns virtual threads l + 32k (k = 0..7); the sum is in lane 0.  The
// first 256 terms are not added (to +0) but are the partial sums, and neither
// the second terms' adds nor the tree's first level run for slots that hold
// none: of 28 warp-wide adds for a row of 275 terms, 12 are left.
// PRE: the ids of the next 256 terms are loaded behind the gathers of these
// (few warps, where the latency of the two loads counts; 8 more registers).
// The loads of 256 terms and more stand under one branch: a predicate each kept
// them from being in flight together (R-MAT 2^16 launched, us: 34 so, 19 now).
// mid_lane_sums: the partial sums of virtual threads 0 .. 31 (after the halving
// tree's first three levels), one per lane.
template <class V, bool COH, bool SOFT, bool PRE>
__device__ __forceinline__ V mid_lane_sums(const V* c, const uint32_t* __restrict__ ed, uint32_t d, uint32_t lane,
                                           bool& bad) {
  V ps[8];
  uint32_t u[8];
  auto ids = [&](uint32_t base) {
    if (base + 256 <= d) {
#pragma unroll
      for (int k = 0; k < 8; ++k) u[k] = __ldg(ed + base + lane + 32u * k);
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) u[k] = base + lane + 32u * k < d ? __ldg(ed + base + lane + 32u * k) : 0u;
    }
  };
  if (PRE) ids(0);
  for (uint32_t base = 0; base < d; base += 256) {
    if (!PRE) ids(base);
    V x[8];
    const bool full = base + 256 <= d;
    if (full) {
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = load_c<COH>(c + u[k]);
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = base + lane + 32u * k < d ? load_c<COH>(c + u[k]) : V(0);
    }
    if (PRE) ids(base + 256);
    if (SOFT) {
#pragma unroll
      for (int k = 0; k < 8; ++k) bad = bad || ((full || base + lane + 32u * k < d) && soft_out_of_range(x[k]));
    }
    if (base == 0) {
#pragma unroll
      for (int k = 0; k < 8; ++k) ps[k] = SOFT ? x[k] : V(0) + x[k];
    } else if (full) {
#pragma unroll
      for (int k = 0; k < 8; k += 2) {
        ps[k] += x[k];
        ps[k + 1] = plus<SOFT>(ps[k + 1], x[k + 1]);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 8; k += 2) {
        if (base + 32u * k < d) ps[k] += x[k];
        if (base + 32u * (k + 1) < d) ps[k + 1] = plus<SOFT>(ps[k + 1], x[k + 1]);
      }
    }
  }
  // halving tree over virtual thread t = lane + 32k; d > 64
  if (d > 128) ps[0] += ps[4];                            // t < 128: += t+128
  if (d > 160) ps[1] = plus<SOFT>(ps[1], ps[5]);
  if (d > 192) ps[2] += ps[6];
  if (d > 224) ps[3] = plus<SOFT>(ps[3], ps[7]);
  ps[0] += ps[2];                                         // t < 64:  += t+64
  ps[1] = plus<SOFT>(ps[1], ps[3]);
  return ps[0] + ps[1];                                   // t < 32:  += t+32
}

// The same by FP64 adds alone, rolled up: it runs on terms out of
// soft_add's range only, and must not add to the sweep's registers.
template <bool COH>
__device__ __forceinline__ double mid_row_sum_plain(const double* c, const uint32_t* __restrict__ ed, uint32_t d,
                                                    uint32_t lane) {
  double ps[8];
#pragma unroll 1
  for (int k = 0; k < 8; ++k) {
    double sum = 0.0;
#pragma unroll 1
    for (uint32_t t = lane + 32u * k; t < d; t += 256) sum += load_c<COH>(c + __ldg(ed + t));
    ps[k] = sum;
  }
#pragma unroll 1
  for (int o = 4; o; o >>= 1)
#pragma unroll 1
    for (int k = 0; k < o; ++k) ps[k] += ps[k + o];
  double x = ps[0];
#pragma unroll 1
  for (int o = 16; o; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  return x;
}
template <class V, bool COH, bool PRE>
__device__ __forceinline__ V mid_row_sum(const V* c, const uint32_t* __restrict__ ed, uint32_t d, uint32_t lane) {
  constexpr bool SOFT = std::is_same<V, double>::value;
  bool bad = false;
  V x = mid_lane_sums<V, COH, SOFT, PRE>(c, ed, d, lane, bad);
  if constexpr (SOFT) {
    if (__any_sync(0xffffffffu, bad)) return mid_row_sum_plain<COH>(c, ed, d, lane);
  }
  x = plus<SOFT>(x, __shfl_down_sync(0xffffffffu, x, 16));
  x += __shfl_down_sync(0xffffffffu, x, 8);
  x = plus<SOFT>(x, __shfl_down_sync(0xffffffffu, x, 4));
  x += __shfl_down_sync(0xffffffffu, x, 2);
  return plus<SOFT>(x, __shfl_down_sync(0xffffffffu, x, 1));
}

// HIGH: the same sum by a block of 256 (thread t of the reference's block);
// part: 256 values of shared memory.  The sum is in thread 0.  Eight gathers are
// in flight, in the last batch too (empty slots add +0.0).  By FP64 adds alone: a
// thread's adds wait for one another, and soft_add's take longer (79 cycles against
// 65).  Static with half of them soft | so, ms: a star of 1M in the cooperative loop
// 13.2 | 9.0, launched 20.3 | 10.8, R-MAT 2^18 with 64 edges a vertex 4.8 | 5.1 (5.2
// and 3.7 once its rows of 1025 to 4096 go by warp).
template <class V, bool COH, bool PRE>
__device__ __forceinline__ V high_thread_sum(const V* c, const uint32_t* __restrict__ ed, uint32_t d, uint32_t t) {
  V acc = V(0);
  uint32_t u[8];
  auto ids = [&](uint32_t base) {
    if (base + 8 * 256 <= d) {
#pragma unroll
      for (int k = 0; k < 8; ++k) u[k] = __ldg(ed + base + 256 * k + t);
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) u[k] = base + 256 * k + t < d ? __ldg(ed + base + 256 * k + t) : 0u;
    }
  };
  if (PRE) ids(0);
  uint32_t base = 0;
  for (; base + 8 * 256 <= d; base += 8 * 256) {
    if (!PRE) ids(base);
    V x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = load_c<COH>(c + u[k]);
    if (PRE) ids(base + 8 * 256);
#pragma unroll
    for (int k = 0; k < 8; ++k) acc += x[k];
  }
  if (base < d) {
    if (!PRE) ids(base);
    V x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = base + 256 * k + t < d ? load_c<COH>(c + u[k]) : V(0);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (base + 256 * k < d) acc += x[k];
  }
  return acc;
}
template <class V, bool COH, bool PRE>
__device__ __forceinline__ V high_row_sum(const V* c, const uint32_t* __restrict__ ed, uint32_t d, uint32_t t, V* part) {
  part[t] = high_thread_sum<V, COH, PRE>(c, ed, d, t);
  __syncthreads();
  if (t < 128) part[t] += part[t + 128];
  __syncthreads();
  if (t < 64) part[t] += part[t + 64];
  __syncthreads();
  V x = V(0);
  if (t < 32) {
    x = part[t] + part[t + 32];
#pragma unroll
    for (int o = 16; o; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  }
  __syncthreads();  // part is free for the next row
  return x;
}

}  // namespace prx
