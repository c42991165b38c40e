// prx_ppr.cu -- batched personalized PageRank: up to 64 teleport vectors per
// column block, solved together.  No counterpart in the reference (its
// solvers take the uniform teleport (1-P)/N only, inc/pagerankCuda.hxx:679).
//
// Vector k teleports uniformly to its seed set S_k:
//   r_k = (1-P) t_k + P * A^T D^-1 r_k,   t_k = (1/|S_k|) sum_{s in S_k} e_s,
// iterated by Jacobi sweeps from r_k = t_k until the L-inf change over all
// vertices and vectors of one sweep is below the tolerance (the reference's
// convergence test, :680,689, taken over the whole block).
//
// Layout: ranks are vertex-major, C values per vertex, where C is the smallest
// of 8, 16, 24, 32, 48 and 64 that holds the block's vectors.  A lane owns 16
// bytes of a row (three columns, strided, for 24 and 48), so a row is a
// coalesced gather by 2 to 32 lanes, and a warp works on 1 to 16 vertices side
// by side.
// Contributions are not stored: each gathered row is scaled by the source's
// reciprocal out-degree in the fma.
//
// What bounds the sweeps: the FP64 ones GB300's FP64 pipe (16 to 17 cycles a
// warp-wide fma, 93% busy), the FP32 ones the way from L2 (about 10 TB/s).
// Measured, us a sweep, 64 columns with a vertex per warp and a block per
// 512-edge segment | so: R-MAT 2^20, 64 vectors, FP32 914 | 790; R-MAT 2^18, 64
// vectors, FP64 760 | 643; web-like 200k, 24 vectors, FP64 895 | 370, 10
// vectors, FP32 240 | 94, 64 vectors, FP32 253 | 251.
//
// Precision:
//  - PRX_FP64: FP64 rows, FP64 sums.
//  - PRX_FP32_REFINE: defect correction as for the static solver -- an FP64
//    residual sweep from the FP64 base x (rho = C + P A^T D^-1 x - x, its
//    L-inf the convergence test), then FP32 sweeps of the correction
//    e' = rho + P A^T D^-1 e (FP32 rows, half the bytes), then x += e.  The
//    FP32 sweeps of a round stop when their change is below the tolerance or
//    below 2^-18 of the correction's size (FP32 cannot resolve more), or at
//    the iteration cap.
//
// Rows of in-degree up to low_max (64 by default): a row's lanes per vertex.
// Longer rows are cut into segments of `seg` in-edges (512 by default) of
// eight contiguous parts; a part's sum is a partial row, and a second kernel
// adds a segment's parts, and a vertex's segments, in order and finishes the
// vertex.  Where memory for the parts' partial rows or for the FP32 sweeps'
// pairs is short, a segment's parts are summed one after the other and ids are
// read instead: the same bits, slower.  Every sum has a fixed order for given low_max / seg,
// so results are deterministic; prx_autotune_ppr picks both per graph.
//
// Loop: by default the whole iteration loop of a column block is one CUDA
// graph launch -- a conditional WHILE node over FP64 sweeps, and for the
// refinement a nested WHILE node over the FP32 correction sweeps of each
// round -- whose condition kernels read the device control block, so the
// host waits once per block; prx_options.loop = PRX_LOOP_HOST runs the same
// kernels from a host loop that reads the control block back between batches
// of sweeps.  Both run the same kernels in the same order (same results).
#include <algorithm>
#include <type_traits>
#include <vector>
#include "prx_ctx.h"
#include "prx_device.cuh"

namespace prx {

constexpr int kCols = 64;         // vectors per column block at most
constexpr uint32_t kSeg = 512;    // default in-edges per segment of a long row
constexpr uint32_t kSegParts = 8; // parts of a segment, summed side by side
constexpr uint32_t kSpread = 4;   // segments of a row past which blocks combine it
constexpr uint32_t kSlice = 8;    // lanes of a row that such a block takes

enum PprMode { PPR_J64 = 0, PPR_R64 = 1, PPR_S32 = 2 };

struct PprWs {
  int device = 0;
  uint32_t n = 0;                 // vertices the row buffers hold
  bool has32 = false;
  double* x[2] = {nullptr, nullptr};   // FP64 ranks, [n][64], ping-pong (refinement: base, sweep output)
  float* rho = nullptr;                // FP32 refinement: residual [n][64]
  float* e[2] = {nullptr, nullptr};    // FP32 corrections, ping-pong
  double* part = nullptr;              // partial rows of the long rows' parts (or segments) [nparts][C]
  size_t part_cap = 0;
  uint2* parts = nullptr;              // vertex, first edge
  size_t parts_cap = 0;
  uint32_t* partstart = nullptr;       // first part of each long vertex (+ total), PprArgs::longs
  size_t partstart_cap = 0;
  uint32_t* big = nullptr;             // vertices above a low_max other than 64, and their scan
  size_t big_cap = 0;
  uint32_t* toff = nullptr;            // teleport entries by vertex: offsets (n+1)
  uint32_t* tent = nullptr;            // entries: vertex, column (sorted)
  double* tmass = nullptr;             // entry mass 1/|S_k|
  size_t t_cap = 0, tm_cap = 0;
  double* out = nullptr;               // device staging of the host output
  size_t out_cap = 0;
};

void ppr_free(PprWs* w) {
  if (!w) return;
  cudaSetDevice(w->device);
  for (int i = 0; i < 2; ++i) {
    cudaFree(w->x[i]);
    cudaFree(w->e[i]);
  }
  cudaFree(w->rho);
  cudaFree(w->part);
  cudaFree(w->parts);
  cudaFree(w->partstart);
  cudaFree(w->big);
  cudaFree(w->toff);
  cudaFree(w->tent);
  cudaFree(w->tmass);
  cudaFree(w->out);
  delete w;
}

struct PprArgs {
  const uint32_t* xtoff;
  const unsigned long long* xtbase;  // row segments (see GraphDev); null: one segment
  uint32_t seg_shift;
  const double* rcp;
  const float* rcp32;
  const uint32_t* xtedg;
  const uint2* pair;              // per in-edge, laid out like xtedg: source, bits of its FP32 reciprocal out-degree
                                  // (FP32 sweeps; null: no memory for it, they read ids and gather reciprocals)
  const uint32_t* toff;
  const uint32_t* tcol;           // column of each teleport entry
  const double* tmass;
  double* x[2];
  float* rho;
  float* e[2];
  const uint32_t* big;            // vertices with in-degree > low_max
  uint32_t nbig;
  uint32_t low_max;               // rows up to this in-degree are summed whole, LPR lanes per vertex
  uint32_t seg;                   // in-edges per segment of a longer row (a multiple of kSegParts)
  uint32_t per;                   // in-edges per part: seg / kSegParts
  uint32_t group;                 // partial rows a segment: kSegParts, or 1 when there is no memory for its parts'
  const uint32_t* partstart;      // [nbig + 1]: each long row's first partial row
  const uint2* parts;             // vertex, first edge (relative to its row segment)
  uint32_t nparts;
  const uint32_t* longs;          // positions in big of the rows of more than spread partial rows
  uint32_t nlong, spread;
  double* part;                   // the partial rows
  State* st;
  uint32_t n;
  const uint32_t* rows;           // the vertices of the short rows in the order they are taken (null: by id)
  uint32_t nrows;
  uint32_t batch;                 // vertices of a unit, whose bounds a warp loads at once (at most 32)
  int cols;                       // C: columns stored per vertex
  bool share;                     // a fixed share of the units per warp
  bool flat;                      // 64 columns: the short rows by k_ppr_flat
  double P, Q;                    // damping, 1 - damping
  float P32;                      // (float)P: a conversion in the kernel runs on the FP64 pipe
};

template <int MODE> struct PprType { using S = double; };
template <> struct PprType<PPR_S32> { using S = float; };

// How a warp holds rows of C columns: LPR lanes per row, G rows side by side,
// N columns per lane -- columns N sub .. N sub + N - 1 of lane sub, read as one
// 16-byte vector, or (VEC false) columns sub + LPR i.
template <int MODE, int C> struct PprShape {
  using S = typename PprType<MODE>::S;
  static constexpr bool VEC = C % 3 != 0;
  static constexpr int N = VEC ? 16 / (int)sizeof(S) : 3;
  static constexpr int LPR = C / N;
  static constexpr int G = 32 / LPR;
  static constexpr int U = 4;       // rows a lane has in flight (ppr_gather's branches are for four)
  static constexpr int BLOCKS = 4;  // resident blocks of 256 per SM
  using Raw = typename std::conditional<sizeof(S) == 8, double2, float4>::type;
  struct V {
    S c[N];
    __device__ __forceinline__ S& operator[](int i) { return c[i]; }
    __device__ __forceinline__ S operator[](int i) const { return c[i]; }
  };
  static_assert(LPR * G == 32, "a warp's lanes");
  // row r of an array of rows, this lane's columns; LDG: by the read-only path
  template <bool LDG>
  __device__ static __forceinline__ V load(const S* rows, size_t r, uint32_t sub) {
    V x;
    if constexpr (VEC) {
      const Raw* at = reinterpret_cast<const Raw*>(rows) + r * LPR + sub;
      const Raw y = LDG ? __ldg(at) : *at;
      x[0] = y.x;
      x[1] = y.y;
      if constexpr (N == 4) {
        x[2] = y.z;
        x[3] = y.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) x[i] = LDG ? __ldg(rows + r * C + sub + LPR * i) : rows[r * C + sub + LPR * i];
    }
    return x;
  }
  __device__ static __forceinline__ void store(S* rows, size_t r, uint32_t sub, const V& x) {
    if constexpr (VEC) {
      Raw y;
      y.x = x[0];
      y.y = x[1];
      if constexpr (N == 4) {
        y.z = x[2];
        y.w = x[3];
      }
      reinterpret_cast<Raw*>(rows)[r * LPR + sub] = y;
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) rows[r * C + sub + LPR * i] = x[i];
    }
  }
  // the lane's i-th column
  __device__ static __forceinline__ uint32_t column(uint32_t sub, int i) { return VEC ? sub * N + i : sub + LPR * i; }
};

template <int MODE>
__device__ __forceinline__ bool ppr_skip(const State* st) {
  return st->done || (MODE == PPR_S32 && st->inner_done);
}

// Source rows of this sweep.
template <int MODE>
__device__ __forceinline__ const typename PprType<MODE>::S* ppr_src(const PprArgs& a, const State* st) {
  if constexpr (MODE == PPR_J64) return a.x[st->iter & 1];
  else if constexpr (MODE == PPR_R64) return a.x[0];
  else return a.e[st->k32 & 1];
}
// An in-edge as a sweep reads it, by all lanes of its row at once: with PAIRS
// (the FP32 sweeps, which the L1 bounds) the source and the bits of its FP32
// reciprocal, half the wavefronts of an id, a reciprocal gather and the row;
// else the source's id.
template <bool PAIRS> struct PprEdge {
  using T = uint32_t;
  __device__ static __forceinline__ const T* base(const PprArgs& a) { return a.xtedg; }
  __device__ static __forceinline__ T none() { return 0; }
  __device__ static __forceinline__ uint32_t source(T e) { return e; }
};
template <> struct PprEdge<true> {
  using T = uint2;
  __device__ static __forceinline__ const T* base(const PprArgs& a) { return a.pair; }
  __device__ static __forceinline__ T none() { return make_uint2(0, 0); }
  __device__ static __forceinline__ uint32_t source(T e) { return e.x; }
};
// The reciprocals of a mode's precision.
template <int MODE>
__device__ __forceinline__ const typename PprType<MODE>::S* ppr_rcp(const PprArgs& a) {
  if constexpr (MODE == PPR_S32) return a.rcp32;
  else return a.rcp;
}
// acc += row(u) / outdeg(u) over the len edges at ed, by the LPR lanes of a row
// (every lane of the warp calls it; rows may differ in length), one edge after
// the other.  pr: the first U edges, loaded by the caller (ppr_edges).  Up to U
// rows are in flight.
template <int MODE, int C, bool PAIRS, class T>
__device__ __forceinline__ void ppr_edges(const T* __restrict__ ed, uint32_t len, T pr[PprShape<MODE, C>::U]) {
#pragma unroll
  for (int k = 0; k < PprShape<MODE, C>::U; ++k) pr[k] = (uint32_t)k < len ? __ldg(ed + k) : PprEdge<PAIRS>::none();
}
template <int MODE, int C, bool PAIRS, class T>
__device__ __forceinline__ void ppr_gather(const typename PprType<MODE>::S* __restrict__ src,
                                           const typename PprType<MODE>::S* __restrict__ rcp,
                                           const T* __restrict__ ed, uint32_t len, T pr[PprShape<MODE, C>::U],
                                           uint32_t sub, typename PprShape<MODE, C>::V& acc) {
  using Sh = PprShape<MODE, C>;
  using S = typename Sh::S;
  using V = typename Sh::V;
  constexpr int U = PprShape<MODE, C>::U;
  const uint32_t longest = Sh::G == 1 ? len : __reduce_max_sync(0xffffffffu, len);
  for (uint32_t base = 0; base < longest; base += U) {
    V g[U];
    S w[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (base + k < len) {
        const uint32_t u = PprEdge<PAIRS>::source(pr[k]);
        g[k] = Sh::template load<true>(src, u, sub);
        if constexpr (PAIRS) w[k] = __uint_as_float(pr[k].y);
        else w[k] = __ldg(rcp + u);
      } else {  // + 0 * 0 leaves the sum
#pragma unroll
        for (int i = 0; i < Sh::N; ++i) g[k][i] = S(0);
        w[k] = S(0);
      }
    }
    if (base + U < longest) ppr_edges<MODE, C, PAIRS>(ed + base + U, len > base + U ? len - base - U : 0u, pr);
    auto add = [&](int k) {
#pragma unroll
      for (int i = 0; i < Sh::N; ++i) acc[i] = fma(g[k][i], w[k], acc[i]);
    };
    if constexpr (MODE == PPR_S32) {
#pragma unroll
      for (int k = 0; k < U; ++k) add(k);
    } else {
      // an FP64 fma issued for no row costs as much as one: branches, not
      // predicates, over the rows the warp has
      const uint32_t n = longest - base;
      if (n >= 4) {
#pragma unroll
        for (int k = 0; k < 4; ++k) add(k);
      } else {
        switch (n) {
          case 1: add(0); break;
          case 2: add(0); add(1); break;
          default: add(0); add(1); add(2); break;
        }
      }
    }
  }
}

// Finish vertex v from its gathered sum (sub: which 16 bytes of the row);
// returns the lane's L-inf term (bits of a double, or of a float for PPR_S32)
// and, for PPR_S32, the size of the new correction in *emag.
template <int MODE, int C>
__device__ __forceinline__ unsigned long long ppr_finish(const PprArgs& a, const State* st, uint32_t v,
                                                         const typename PprShape<MODE, C>::V& acc, uint32_t sub,
                                                         unsigned int* emag) {
  using Sh = PprShape<MODE, C>;
  using V = typename Sh::V;
  if constexpr (MODE == PPR_S32) {
    const int q = st->k32 & 1;
    const V r = Sh::template load<false>(a.rho, v, sub), old = Sh::template load<false>(a.e[q], v, sub);
    V en;
    const float P = a.P32;
    float big = 0.f, chg = 0.f;
#pragma unroll
    for (int i = 0; i < Sh::N; ++i) {
      en[i] = fmaf(P, acc[i], r[i]);
      big = fmaxf(big, fabsf(en[i]));
      chg = fmaxf(chg, fabsf(en[i] - old[i]));
    }
    Sh::store(a.e[q ^ 1], v, sub, en);
    *emag = __float_as_uint(big);
    return __float_as_uint(chg);
  } else {
    const int p = MODE == PPR_J64 ? (st->iter & 1) : 0;
    const V old = Sh::template load<false>(a.x[p], v, sub);
    V t;
#pragma unroll
    for (int i = 0; i < Sh::N; ++i) t[i] = 0.0;
    const uint32_t t0 = __ldg(a.toff + v), t1 = __ldg(a.toff + v + 1);
    if (t0 < t1) {  // few vertices are seeds; Q * 0 is 0
      for (uint32_t i = t0; i < t1; ++i) {
        const uint32_t col = __ldg(a.tcol + i);
#pragma unroll
        for (int k = 0; k < Sh::N; ++k)
          if (col == Sh::column(sub, k)) t[k] += __ldg(a.tmass + i);
      }
#pragma unroll
      for (int i = 0; i < Sh::N; ++i) t[i] = a.Q * t[i];
    }
    V an;
    unsigned long long chg = 0;  // |change| as bits (non-negative doubles order as their bits)
    float r[Sh::N];
#pragma unroll
    for (int i = 0; i < Sh::N; ++i) {
      an[i] = fma(a.P, acc[i], t[i]);
      const double d = an[i] - old[i];
      if (MODE == PPR_R64) r[i] = (float)d;
      const unsigned long long b = dbits(d) & ~(1ull << 63);
      chg = b > chg ? b : chg;
    }
    Sh::store(a.x[p ^ 1], v, sub, an);
    if constexpr (MODE == PPR_R64 && Sh::VEC) {
      const float2 r2 = make_float2(r[0], r[1]);
      reinterpret_cast<float2*>(a.rho)[(size_t)v * Sh::LPR + sub] = r2;
      reinterpret_cast<float2*>(a.e[0])[(size_t)v * Sh::LPR + sub] = r2;
    } else if constexpr (MODE == PPR_R64) {
#pragma unroll
      for (int i = 0; i < Sh::N; ++i) {
        const size_t at = (size_t)v * C + Sh::column(sub, i);
        a.rho[at] = r[i];
        a.e[0][at] = r[i];
      }
    }
    return chg;
  }
}

template <int MODE>
__device__ __forceinline__ void ppr_reduce(State* st, unsigned long long dmax, unsigned int emag) {
  if constexpr (MODE == PPR_S32) {
    block_max_u32((unsigned int)dmax, &st->el32_bits[st->k32 & 1]);
    block_max_u32(emag, &st->e32max_bits[st->k32 & 1]);
  } else {
    block_max_bits(dmax, &st->el_bits[st->iter & 1]);
  }
}

// One sweep's rows.  A warp takes units: first G parts of long rows (partial
// sums of a.per in-edges each, added up by k_ppr_combine), then batches of
// short rows (in-degree <= low_max), LPR lanes per vertex and G vertices side
// by side; a batch's bounds are loaded by a lane each, and the first edges of
// the next G vertices while it sums these.  No warp waits for another.
template <int MODE, int C, bool PAIRS>
__global__ void __launch_bounds__(256, PprShape<MODE, C>::BLOCKS) k_ppr_rows(PprArgs a) {
  using Ed = PprEdge<PAIRS>;
  using Sh = PprShape<MODE, C>;
  using S = typename Sh::S;
  using V = typename Sh::V;
  constexpr uint32_t LPR = Sh::LPR, G = Sh::G;
  constexpr int U = Sh::U;
  State* st = a.st;
  if (ppr_skip<MODE>(st)) return;
  const S* __restrict__ src = ppr_src<MODE>(a, st);
  const S* __restrict__ rcp = ppr_rcp<MODE>(a);
  const uint32_t lane = lane_id(), sub = lane % LPR, grp = lane / LPR;
  unsigned long long dmax = 0;
  unsigned int emag = 0;
  const uint32_t nb = (uint32_t)(((uint64_t)a.nrows + a.batch - 1) / a.batch);
  const uint32_t np = (a.nparts + G - 1) / G;
  auto zero = [](V& x) {
#pragma unroll
    for (int k = 0; k < Sh::N; ++k) x[k] = S(0);
  };
  // units are taken from a counter (reset by the sweep's finalize kernel), the
  // next one while this one is summed: they differ in length and in what the
  // caches hold, and a fixed share per warp left a seventh of the warps idle
  // (with few units the counter's latency is what counts: a.share)
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  uint32_t next = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  auto take = [&] {
    if (a.share) next += warps;
    else if (lane == 0) next = atomicAdd(&st->work, 1u);
  };
  if (!a.share) take();
  typename Ed::T pr[U];
  for (;;) {
    const uint32_t b = __shfl_sync(0xffffffffu, next, 0);
    if (b >= np + nb) break;
    take();
    if (b < np) {
      const uint32_t i = b * G + grp;
      uint32_t len = 0;
      const typename Ed::T* ed = Ed::base(a);
      if (i < a.nparts) {
        const uint2 w = __ldg(a.parts + i);  // vertex, first edge
        const uint32_t end = __ldg(a.xtoff + seg_index(w.x, a.seg_shift) + 1);
        len = min(a.per, end - w.y);
        ed += w.y + (a.xtbase ? a.xtbase[(uint64_t)w.x >> a.seg_shift] : 0ull);
      }
      ppr_edges<MODE, C, PAIRS>(ed, len, pr);
      V acc;
      zero(acc);
      ppr_gather<MODE, C, PAIRS>(src, rcp, ed, len, pr, sub, acc);
      if (i < a.nparts) Sh::store(reinterpret_cast<S*>(a.part), i, sub, acc);
      continue;
    }
    const uint32_t i0 = (b - np) * a.batch;
    // lane i: vertex i of the batch (len 0xffffffff: none, or a long row)
    uint32_t mv = 0, ml = 0xffffffffu;
    unsigned long long ms = 0;
    if (lane < a.batch && i0 + lane < a.nrows) {
      mv = a.rows ? __ldg(a.rows + i0 + lane) : i0 + lane;
      const uint64_t iv = seg_index(mv, a.seg_shift);
      const uint32_t s = __ldg(a.xtoff + iv), len = __ldg(a.xtoff + iv + 1) - s;
      ms = s + (a.xtbase ? a.xtbase[(uint64_t)mv >> a.seg_shift] : 0ull);
      if (len <= a.low_max) ml = len;
    }
    const uint32_t cnt = min(a.batch, a.nrows - i0);
    uint32_t v, len;
    const typename Ed::T* ed;
    auto fetch = [&](uint32_t i) {  // vertex i + grp of the batch and its first edges
      const uint32_t k = i + grp;
      v = __shfl_sync(0xffffffffu, mv, k & 31);
      ed = Ed::base(a) + __shfl_sync(0xffffffffu, ms, k & 31);
      len = __shfl_sync(0xffffffffu, ml, k & 31);
      if (k >= cnt) len = 0xffffffffu;
      ppr_edges<MODE, C, PAIRS>(ed, len == 0xffffffffu ? 0u : len, pr);
    };
    fetch(0);
    for (uint32_t i = 0; i < cnt; i += G) {
      const uint32_t cv = v, cl = len;
      V acc;
      zero(acc);
      ppr_gather<MODE, C, PAIRS>(src, rcp, ed, cl == 0xffffffffu ? 0u : cl, pr, sub, acc);
      if (i + G < cnt) fetch(i + G);
      if (cl == 0xffffffffu) continue;
      unsigned int em = 0;
      const unsigned long long d = ppr_finish<MODE, C>(a, st, cv, acc, sub, &em);
      dmax = d > dmax ? d : dmax;
      emag = em > emag ? em : emag;
    }
  }
  ppr_reduce<MODE>(st, dmax, emag);
}

// The short rows of a 64-column sweep, a warp per vertex in id order, two
// columns per lane: 32 registers (FP32), so 64 warps an SM, and 4-byte ids
// (their reciprocals hit the L1), which web-like graphs -- rows of one length,
// bound by the L1 and the way to it, or by the FP64 pipe with nothing to gain
// from a better order -- need more than the side-by-side rows: FP32 174 against
// 192 us a sweep on 200k vertices, FP64 the
// 32 registers matter too: 60 vectors on 93k vertices 11.42 against 11.48 ms.  The same sums.
template <int MODE>
__global__ void __launch_bounds__(256) k_ppr_flat(PprArgs a) {
  using S = typename PprType<MODE>::S;
  using V2 = typename std::conditional<MODE == PPR_S32, float2, double2>::type;
  State* st = a.st;
  if (ppr_skip<MODE>(st)) return;
  const V2* __restrict__ src = reinterpret_cast<const V2*>(ppr_src<MODE>(a, st));
  const S* __restrict__ rc = ppr_rcp<MODE>(a);
  const uint32_t lane = lane_id(), warps = (gridDim.x * blockDim.x) >> 5;
  unsigned long long dmax = 0;
  unsigned int emag = 0;
  for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < a.n; v += warps) {
    const uint64_t iv = seg_index(v, a.seg_shift);
    const uint32_t s = __ldg(a.xtoff + iv), e = __ldg(a.xtoff + iv + 1);
    if (e - s > a.low_max) continue;
    const uint32_t* __restrict__ edg = seg_edges(a.xtedg, a.xtbase, a.seg_shift, v);
    V2 acc;
    acc.x = acc.y = S(0);
    uint32_t j = s;
    for (; j + 4 <= e; j += 4) {
      const uint32_t u0 = __ldg(edg + j), u1 = __ldg(edg + j + 1), u2 = __ldg(edg + j + 2), u3 = __ldg(edg + j + 3);
      const V2 g0 = __ldg(src + (size_t)u0 * 32 + lane), g1 = __ldg(src + (size_t)u1 * 32 + lane);
      const V2 g2 = __ldg(src + (size_t)u2 * 32 + lane), g3 = __ldg(src + (size_t)u3 * 32 + lane);
      const S y0 = __ldg(rc + u0), y1 = __ldg(rc + u1), y2 = __ldg(rc + u2), y3 = __ldg(rc + u3);
      acc.x = fma(g0.x, y0, acc.x); acc.y = fma(g0.y, y0, acc.y);
      acc.x = fma(g1.x, y1, acc.x); acc.y = fma(g1.y, y1, acc.y);
      acc.x = fma(g2.x, y2, acc.x); acc.y = fma(g2.y, y2, acc.y);
      acc.x = fma(g3.x, y3, acc.x); acc.y = fma(g3.y, y3, acc.y);
    }
    for (; j < e; ++j) {
      const uint32_t u = __ldg(edg + j);
      const V2 g = __ldg(src + (size_t)u * 32 + lane);
      const S y = __ldg(rc + u);
      acc.x = fma(g.x, y, acc.x);
      acc.y = fma(g.y, y, acc.y);
    }
    if constexpr (MODE == PPR_S32) {
      const int q = st->k32 & 1;
      const size_t at = (size_t)v * 32 + lane;
      const float2 r = reinterpret_cast<const float2*>(a.rho)[at], old = src[at];
      const float P = a.P32;
      const float2 en = make_float2(fmaf(P, acc.x, r.x), fmaf(P, acc.y, r.y));
      reinterpret_cast<float2*>(a.e[q ^ 1])[at] = en;
      emag = max(emag, __float_as_uint(fmaxf(fabsf(en.x), fabsf(en.y))));
      dmax = max(dmax, (unsigned long long)__float_as_uint(fmaxf(fabsf(en.x - old.x), fabsf(en.y - old.y))));
    } else {
      // ppr_finish for two columns, in the 32 registers that the sum has
      const size_t at = (size_t)v * 32 + lane;
      double tx = 0.0, ty = 0.0;
      for (uint32_t i = __ldg(a.toff + v), ie = __ldg(a.toff + v + 1); i < ie; ++i) {
        const uint32_t col = __ldg(a.tcol + i);
        if ((col >> 1) == lane) {
          if (col & 1u) ty += __ldg(a.tmass + i);
          else tx += __ldg(a.tmass + i);
        }
      }
      const double2 an = make_double2(fma(a.P, acc.x, a.Q * tx), fma(a.P, acc.y, a.Q * ty));
      const int p = MODE == PPR_J64 ? (st->iter & 1) : 0;
      const double2 old = reinterpret_cast<const double2*>(a.x[p])[at];
      reinterpret_cast<double2*>(a.x[p ^ 1])[at] = an;
      const double dx = an.x - old.x, dy = an.y - old.y;
      if (MODE == PPR_R64) {
        const float2 r = make_float2((float)dx, (float)dy);
        reinterpret_cast<float2*>(a.rho)[at] = r;
        reinterpret_cast<float2*>(a.e[0])[at] = r;
      }
      const unsigned long long d = dbits(fmax(fabs(dx), fabs(dy)));
      dmax = d > dmax ? d : dmax;
    }
  }
  ppr_reduce<MODE>(st, dmax, emag);
}

// The long rows' segments without memory for their parts' partial rows (a.group
// 1): a row's lanes sum a segment's parts one after the other and add them up as
// k_ppr_combine would, the same bits, and leave one partial row a segment.
template <int MODE, int C>
__global__ void __launch_bounds__(256) k_ppr_segments(PprArgs a) {
  using Sh = PprShape<MODE, C>;
  using S = typename Sh::S;
  using V = typename Sh::V;
  State* st = a.st;
  if (ppr_skip<MODE>(st)) return;
  const S* __restrict__ src = ppr_src<MODE>(a, st);
  const S* __restrict__ rcp = ppr_rcp<MODE>(a);
  const uint32_t lane = lane_id(), sub = lane % Sh::LPR, grp = lane / Sh::LPR;
  for (uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < (a.nparts + Sh::G - 1) / Sh::G;
       b += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t i = b * Sh::G + grp;
    uint32_t rest = 0;  // edges of the segment left
    const uint32_t* ed = a.xtedg;
    if (i < a.nparts) {
      const uint2 w = __ldg(a.parts + i);  // vertex, first edge
      rest = min(a.seg, __ldg(a.xtoff + seg_index(w.x, a.seg_shift) + 1) - w.y);
      ed += w.y + (a.xtbase ? a.xtbase[(uint64_t)w.x >> a.seg_shift] : 0ull);
    }
    V acc;
#pragma unroll 1
    for (uint32_t q = 0; q < kSegParts; ++q) {
      const uint32_t len = min(a.per, rest);
      uint32_t pr[Sh::U];
      V x;
#pragma unroll
      for (int k = 0; k < Sh::N; ++k) x[k] = S(0);
      ppr_edges<MODE, C, false>(ed, len, pr);
      ppr_gather<MODE, C, false>(src, rcp, ed, len, pr, sub, x);
#pragma unroll
      for (int k = 0; k < Sh::N; ++k) acc[k] = q == 0 ? x[k] : (len ? acc[k] + x[k] : acc[k]);
      ed += len;
      rest -= len;
    }
    if (i < a.nparts) Sh::store(reinterpret_cast<S*>(a.part), i, sub, acc);
  }
}

// Long rows: a row's lanes per vertex add its segments in order, a segment
// being its GROUP parts (fewer in the last) added in order: kSegParts, or one
// partial row that holds their sum.  Of rows of more than a.spread partial rows
// (a.longs) the first blocks take kSlice lanes' columns each: their groups of
// lanes form segments side by side and leave them in shared memory to the first
// group, which adds them in the same order.  Solves, ms, every row by a group of
// lanes | so, of 5 vectors in FP32, 40 in FP32 and 64 in FP64: R-MAT 2^19 8.3 | 5.3,
// 18.2 | 15.3, 57.1 | 54.2; 100 hubs of 15,000 1.85 | 0.90, 2.56 | 1.84, 5.09 | 4.51;
// a star of 64k 3.69 | 0.91, 3.67 | 1.36, 4.92 | 2.31.  With the line at 8 | 16
// segments (5 vectors) R-MAT 2^19 5.4 | 5.4, 2^17 2.1 | 2.5.
template <int MODE, int C, uint32_t GROUP>
__global__ void __launch_bounds__(256) k_ppr_combine(PprArgs a, uint32_t long_blocks) {
  using Sh = PprShape<MODE, C>;
  using S = typename Sh::S;
  using V = typename Sh::V;
  constexpr uint32_t LPR = Sh::LPR;
  constexpr uint32_t SLICE = LPR < kSlice ? LPR : kSlice, SLICES = LPR / SLICE, SEGS = 256 / SLICE - 1;
  State* st = a.st;
  if (ppr_skip<MODE>(st)) return;
  const S* part = reinterpret_cast<const S*>(a.part);
  uint32_t sub = threadIdx.x % LPR;
  unsigned long long dmax = 0;
  unsigned int emag = 0;
  auto segment = [&](uint32_t g, uint32_t end) {  // the sum of partial rows g .. g + GROUP - 1 (g < end)
    V x[GROUP];
#pragma unroll
    for (uint32_t k = 0; k < GROUP; ++k) {
      if (g + k < end) {
        x[k] = Sh::template load<false>(part, g + k, sub);
      } else {
#pragma unroll
        for (int j = 0; j < Sh::N; ++j) x[k][j] = S(0);
      }
    }
#pragma unroll
    for (uint32_t k = 1; k < GROUP; ++k)
      if (g + k < end) {
#pragma unroll
        for (int j = 0; j < Sh::N; ++j) x[0][j] += x[k][j];
      }
    return x[0];
  };
  auto finish = [&](uint32_t i, const V& acc) {
    unsigned int em = 0;
    const unsigned long long d = ppr_finish<MODE, C>(a, st, a.big[i], acc, sub, &em);
    dmax = d > dmax ? d : dmax;
    emag = em > emag ? em : emag;
  };
  if (blockIdx.x < long_blocks) {
    __shared__ V sums[2][256];
    const uint32_t row = threadIdx.x / SLICE;  // 0: adds the segments, the others form them
    for (uint32_t k = blockIdx.x; k < a.nlong * SLICES; k += long_blocks) {
      const uint32_t i = a.longs[k / SLICES], end = a.partstart[i + 1];
      sub = k % SLICES * SLICE + threadIdx.x % SLICE;
      V acc;
#pragma unroll
      for (int j = 0; j < Sh::N; ++j) acc[j] = S(0);
      uint32_t b = 0;
      for (uint32_t g = a.partstart[i]; g < end; g += GROUP * SEGS, b ^= 1u) {
        const uint32_t mine = g + (row - 1) * GROUP;
        if (row && mine < end) sums[b][threadIdx.x] = segment(mine, end);
        __syncthreads();  // (b is added up while b ^ 1 is filled)
        if (row == 0) {
          const uint32_t m = min(SEGS, (end - g + GROUP - 1) / GROUP);
#pragma unroll 4
          for (uint32_t q = 1; q <= m; ++q) {
            const V x = sums[b][q * SLICE + threadIdx.x];
#pragma unroll
            for (int j = 0; j < Sh::N; ++j) acc[j] += x[j];
          }
        }
      }
      if (row == 0) finish(i, acc);
      __syncthreads();  // before the next row's first sums
    }
  } else {
    for (uint32_t i = ((blockIdx.x - long_blocks) * blockDim.x + threadIdx.x) / LPR; i < a.nbig;
         i += (gridDim.x - long_blocks) * blockDim.x / LPR) {
      const uint32_t end = a.partstart[i + 1], start = a.partstart[i];
      if (end - start > a.spread) continue;
      V acc;
#pragma unroll
      for (int k = 0; k < Sh::N; ++k) acc[k] = S(0);
      for (uint32_t g = start; g < end; g += GROUP) {
        const V x = segment(g, end);
#pragma unroll
        for (int k = 0; k < Sh::N; ++k) acc[k] += x[k];
      }
      finish(i, acc);
    }
  }
  ppr_reduce<MODE>(st, dmax, emag);
}

// ---- loop control ------------------------------------------------------------
__global__ void k_ppr_fin64(State* st) {  // Jacobi FP64 sweep
  if (st->done) return;
  st->work = 0;
  const int p = st->iter & 1;
  const double el = __longlong_as_double((long long)st->el_bits[p]);
  st->last_delta = el;
  st->iter += 1;
  st->el_bits[p ^ 1] = 0;
  if (el < st->tol || st->iter >= st->max_iter) st->done = 1;
}

__global__ void k_ppr_fin_r64(State* st) {  // refinement: FP64 residual sweep
  if (st->done) return;
  st->work = 0;
  const double el = __longlong_as_double((long long)st->el_bits[st->iter & 1]);
  st->last_delta = el;
  st->iter += 1;
  st->rounds += 1;
  st->el_bits[0] = st->el_bits[1] = 0;
  if (el < st->tol || st->iter >= st->max_iter) {
    st->done = 1;
    return;
  }
  st->k32 = 0;
  st->inner_done = 0;
  st->el32_bits[0] = st->el32_bits[1] = 0;
  st->e32max_bits[0] = st->e32max_bits[1] = 0;
  st->el32_prev[0] = st->el32_prev[1] = 0;
}

__global__ void k_ppr_fin32(State* st) {  // refinement: FP32 correction sweep
  if (st->done || st->inner_done) return;
  st->work = 0;
  const int q = st->k32 & 1;
  const float dl = __uint_as_float(st->el32_bits[q]);
  const float em = __uint_as_float(st->e32max_bits[q]);
  st->iter += 1;
  st->k32 += 1;
  st->el32_bits[q ^ 1] = 0;
  st->e32max_bits[q ^ 1] = 0;
  const float prev = __uint_as_float(st->el32_prev[0]), prev2 = __uint_as_float(st->el32_prev[1]);
  st->el32_prev[1] = st->el32_prev[0];
  st->el32_prev[0] = __float_as_uint(dl);
  if (dl < (float)st->tol || dl < em * 0x1p-18f || st->iter >= st->max_iter ||
      fp32_round_done(dl, prev, prev2, st->tol))
    st->inner_done = 1;
}

// x_b += e (the correction of the last FP32 sweep); nothing once the solve
// is done (the graph loop reaches it after a converged FP64 sweep).
__global__ void k_ppr_commit(PprArgs a) {
  if (a.st->done) return;
  const float* __restrict__ e = a.e[a.st->k32 & 1];
  const size_t total = (size_t)a.n * a.cols;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x)
    a.x[0][i] += (double)e[i];
}

// Conditions of the graph-launched loops.  Each counts its own bodies and
// stops after `cap` of them whatever the other kernels did, so the loops end
// even if a finalize kernel never ran.
__global__ void k_ppr_cond(cudaGraphConditionalHandle h, State* st, int cap, int refine) {
  const int rounds = ++st->graph_rounds;
  const bool more = !st->done && (!refine || st->iter < st->max_iter) && rounds < cap;
  cudaGraphSetConditional(h, more ? 1u : 0u);
}
__global__ void k_ppr_arm_inner(cudaGraphConditionalHandle h, State* st) {
  st->graph_inner = 0;
  cudaGraphSetConditional(h, (!st->done && !st->inner_done) ? 1u : 0u);
}
__global__ void k_ppr_cond_inner(cudaGraphConditionalHandle h, State* st, int cap) {
  const int rounds = ++st->graph_inner;
  cudaGraphSetConditional(h, (!st->done && !st->inner_done && rounds < cap) ? 1u : 0u);
}

// ---- setup ---------------------------------------------------------------------
// toff[v] = first teleport entry of v (entries sorted by vertex).
__global__ void k_ppr_toff(const uint32_t* __restrict__ ent_v, uint32_t nent, uint32_t n, uint32_t* __restrict__ toff) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = nent;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (ent_v[mid] < v) lo = mid + 1;
      else hi = mid;
    }
    toff[v] = lo;
  }
}

// x0 = t (rows zeroed before): each vertex adds its own entries.
__global__ void k_ppr_init(PprArgs a) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < a.n; v += gridDim.x * blockDim.x)
    for (uint32_t i = a.toff[v]; i < a.toff[v + 1]; ++i) a.x[0][(size_t)v * a.cols + a.tcol[i]] += a.tmass[i];
}

// Part counts of the long vertices (ceil(indeg / per)), then the parts.
__global__ void k_ppr_partcount(const uint32_t* __restrict__ xtoff, uint32_t shift, const uint32_t* __restrict__ big,
                                uint32_t nbig, uint32_t per, uint32_t most, uint32_t* __restrict__ cnt) {
  uint32_t* longs = cnt + nbig + 1;  // their number, then they, in any order
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nbig; i += gridDim.x * blockDim.x) {
    const uint32_t parts = (row_len(xtoff, shift, big[i]) + per - 1) / per;
    cnt[i] = parts;
    if (parts > most) longs[1 + atomicAdd(longs, 1u)] = i;
  }
}

// Vertices of in-degree above t: flags (n + 1 entries, the last 0) for the
// scan, then the ascending list.
__global__ void k_ppr_bigflags(const uint32_t* __restrict__ xtoff, uint32_t shift, uint32_t n, uint32_t t,
                               uint32_t* __restrict__ f) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += gridDim.x * blockDim.x)
    f[v] = v < n && row_len(xtoff, shift, v) > t ? 1u : 0u;
}
__global__ void k_ppr_biglist(const uint32_t* __restrict__ xtoff, uint32_t shift, uint32_t n, uint32_t t,
                              const uint32_t* __restrict__ pos, uint32_t* __restrict__ big) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    if (row_len(xtoff, shift, v) > t) big[pos[v]] = v;
}

// A warp per long vertex writes its parts.
__global__ void k_ppr_partfill(const uint32_t* __restrict__ xtoff, uint32_t shift, const uint32_t* __restrict__ big,
                               uint32_t nbig, uint32_t per, const uint32_t* __restrict__ start,
                               uint2* __restrict__ parts) {
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nbig; i += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t v = big[i], g0 = start[i], n = start[i + 1] - g0;
    const uint32_t s0 = xtoff[seg_index(v, shift)];
    for (uint32_t k = lane_id(); k < n; k += 32) parts[g0 + k] = make_uint2(v, s0 + k * per);
  }
}

__global__ void k_ppr_pairs(const uint32_t* __restrict__ edg, uint64_t slots, uint32_t n,
                            const float* __restrict__ rcp32, uint2* __restrict__ pair) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < slots; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t u = edg[i];  // the slots between row segments hold no edge
    pair[i] = make_uint2(u, u < n ? __float_as_uint(__ldg(rcp32 + u)) : 0u);
  }
}

// out[v * nvec + c0 + k] = x[v][k] for k < w (x has cols columns).
__global__ void k_ppr_out(const double* __restrict__ x, uint32_t n, uint32_t cols, uint32_t nvec, uint32_t c0,
                          uint32_t w, double* __restrict__ out) {
  const size_t total = (size_t)n * w;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t v = i / w, k = i % w;
    out[v * nvec + c0 + k] = x[v * cols + k];
  }
}

static inline int grid_for(uint64_t work, int threads, int cap) {
  const uint64_t b = (work + threads - 1) / threads;
  return (int)(b < 1 ? 1 : (b < (uint64_t)cap ? b : cap));
}

template <int MODE, int C>
static void ppr_sweep_c(const PprArgs& a, int sms, cudaStream_t s, uint64_t& launches) {
  constexpr uint32_t G = PprShape<MODE, C>::G;
  PprArgs b = a;
  // Vertices per unit: what the last warps wait for, and what the counter is
  // asked for.  FP64 units are long (a 64-column row takes the pipe 32 cycles
  // an edge): four per group of lanes, R-MAT 2^18 738 us a sweep at 16, 643 at
  // four; FP32 ones eight, R-MAT 2^20 784 at 16 vertices, 830 at four.
  b.batch = std::min<uint32_t>(32, (MODE == PPR_S32 ? 8 : 4) * G);
  while (b.batch > G && (uint64_t)a.nrows / b.batch < 2ull * 32 * sms) b.batch /= 2;
  // few units in all: no counter (R-MAT 2^16, 5 vectors: 41 us a sweep, 52 with it)
  b.share = (uint64_t)a.nrows / b.batch + a.nparts / G < 2ull * 32 * sms;
  if (C == 64 && a.flat) {
    k_ppr_flat<MODE><<<grid_for((uint64_t)a.n * 32, 256, sms * 8), 256, 0, s>>>(a);
    ++launches;
    b.nrows = 0;  // the long rows are left
  }
  if (a.nparts && a.group == 1) {
    k_ppr_segments<MODE, C><<<grid_for((uint64_t)a.nparts * (32 / G), 256, sms * 8), 256, 0, s>>>(a);
    ++launches;
    b.nparts = 0;
  }
  const uint64_t units = ((uint64_t)b.nrows + b.batch - 1) / b.batch + (b.nparts + G - 1) / G;
  if (units) {
    const int grid = grid_for(units * 32, 256, sms * PprShape<MODE, C>::BLOCKS);
    if constexpr (MODE == PPR_S32) {
      if (a.pair) k_ppr_rows<MODE, C, true><<<grid, 256, 0, s>>>(b);
      else k_ppr_rows<MODE, C, false><<<grid, 256, 0, s>>>(b);
    } else {
      k_ppr_rows<MODE, C, false><<<grid, 256, 0, s>>>(b);
    }
    ++launches;
  }
  if (a.nparts) {
    const uint32_t lb = std::min<uint32_t>(a.nlong * std::max(1u, 32 / G / kSlice), 8 * sms);
    const int grid = grid_for((uint64_t)a.nbig * (32 / G), 256, sms * 8) + lb;
    if (a.group == 1) k_ppr_combine<MODE, C, 1><<<grid, 256, 0, s>>>(a, lb);
    else k_ppr_combine<MODE, C, kSegParts><<<grid, 256, 0, s>>>(a, lb);
    ++launches;
  }
}

template <int MODE>
static void ppr_sweep(const PprArgs& a, int sms, cudaStream_t s, uint64_t& launches) {
  switch (a.cols) {
    case 8: return ppr_sweep_c<MODE, 8>(a, sms, s, launches);
    case 16: return ppr_sweep_c<MODE, 16>(a, sms, s, launches);
    case 24: return ppr_sweep_c<MODE, 24>(a, sms, s, launches);
    case 32: return ppr_sweep_c<MODE, 32>(a, sms, s, launches);
    case 48: return ppr_sweep_c<MODE, 48>(a, sms, s, launches);
    default: return ppr_sweep_c<MODE, 64>(a, sms, s, launches);
  }
}

}  // namespace prx

// ---- host driver ---------------------------------------------------------------------
template <class T>
static cudaError_t grow(T** p, size_t& cap, size_t want) {
  if (*p && cap >= want) return cudaSuccess;
  cudaFree(*p);
  *p = nullptr;
  cap = 0;
  cudaError_t e = device_alloc(p, sizeof(T) * (want ? want : 1));
  if (e == cudaSuccess) cap = want;
  return e;
}

static int ppr_ws(prx_context* c, uint32_t n, bool fp32) {
  if (!c->ppr) {
    c->ppr = new PprWs();
    c->ppr->device = c->device;
  }
  PprWs& w = *c->ppr;
  if (w.n < n) {
    for (int i = 0; i < 2; ++i) {
      cudaFree(w.x[i]); w.x[i] = nullptr;
      cudaFree(w.e[i]); w.e[i] = nullptr;
    }
    cudaFree(w.rho); w.rho = nullptr;
    cudaFree(w.toff); w.toff = nullptr;
    w.n = 0;
    w.has32 = false;
    const size_t rows = (size_t)n * kCols;
    for (int i = 0; i < 2; ++i) TRY_CUDA_ST(device_alloc(&w.x[i], sizeof(double) * rows));
    TRY_CUDA_ST(device_alloc(&w.toff, sizeof(uint32_t) * ((size_t)n + 1)));
    w.n = n;
  }
  if (fp32 && !w.has32) {
    const size_t rows = (size_t)w.n * kCols;
    cudaFree(w.rho);  // of a call that ended here
    cudaFree(w.e[0]);
    w.rho = w.e[0] = nullptr;
    TRY_CUDA_ST(device_alloc(&w.rho, sizeof(float) * rows));
    for (int i = 0; i < 2; ++i) TRY_CUDA_ST(device_alloc(&w.e[i], sizeof(float) * rows));
    w.has32 = true;
  }
  return PRX_OK;
}

// The partial rows of the long rows a.big: a.group per segment of a.seg edges.
static cudaError_t ppr_parts(prx_context* c, const GraphDev& g, PprArgs& a) {
  PprWs& w = *c->ppr;
  cudaStream_t s = c->stream;
  const uint32_t per = a.seg / a.group;
  a.spread = kSpread * a.group;
  uint32_t* count = w.partstart + a.nbig;  // parts in all, rows of more than a.spread, those rows
  cudaError_t e = cudaMemsetAsync(count + 1, 0, sizeof(uint32_t), s);
  if (e != cudaSuccess) return e;
  k_ppr_partcount<<<grid_for(a.nbig, 256, c->sms * 4), 256, 0, s>>>(g.xtoff, g.seg_shift, a.big, a.nbig, per, a.spread,
                                                                    w.partstart);
  e = exclusive_scan_u32(w.partstart, a.nbig + 1, s);
  if (e != cudaSuccess) return e;
  uint32_t host[2] = {0, 0};
  e = cudaMemcpyAsync(host, count, sizeof host, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  const uint32_t nparts = host[0];
  if (e == cudaSuccess) e = grow(&w.parts, w.parts_cap, (size_t)nparts);
  if (e == cudaSuccess) e = grow(&w.part, w.part_cap, (size_t)nparts * kCols);
  if (e != cudaSuccess) return e;
  k_ppr_partfill<<<grid_for((uint64_t)a.nbig * 32, 256, c->sms * 8), 256, 0, s>>>(g.xtoff, g.seg_shift, a.big, a.nbig,
                                                                                  per, w.partstart, w.parts);
  a.partstart = w.partstart;
  a.longs = count + 2;
  a.nlong = host[1];
  a.parts = w.parts;
  a.nparts = nparts;
  a.part = w.part;
  return cudaGetLastError();
}

// The long rows of graph g (in-degree above a.low_max) and their partial rows
// into the workspace: a part each, or, without memory for those, a segment each.
static int ppr_segments(prx_context* c, const GraphDev& g, PprArgs& a) {
  PprWs& w = *c->ppr;
  cudaStream_t s = c->stream;
  uint32_t nbig = 0;
  if (a.low_max == kLowMax) {  // the graph's MID and HIGH classes
    nbig = g.cls_begin[NCLS] - g.cls_begin[MID];
    a.big = g.cls_list + g.cls_begin[MID];
  } else {
    TRY_CUDA_ST(grow(&w.big, w.big_cap, 2 * ((size_t)g.n + 1)));
    uint32_t* pos = w.big + g.n + 1;
    k_ppr_bigflags<<<grid_for((uint64_t)g.n + 1, 256, c->sms * 16), 256, 0, s>>>(g.xtoff, g.seg_shift, g.n, a.low_max, pos);
    TRY_CUDA_ST(exclusive_scan_u32(pos, g.n + 1, s));
    k_ppr_biglist<<<grid_for(g.n, 256, c->sms * 16), 256, 0, s>>>(g.xtoff, g.seg_shift, g.n, a.low_max, pos, w.big);
    TRY_CUDA_ST(cudaMemcpyAsync(&nbig, pos + g.n, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    TRY_CUDA_ST(cudaStreamSynchronize(s));
    a.big = w.big;
  }
  a.nbig = nbig;
  a.nparts = 0;
  if (!nbig) return PRX_OK;
  TRY_CUDA_ST(grow(&w.partstart, w.partstart_cap, 2 * (size_t)nbig + 2));
  a.group = kSegParts;
  cudaError_t e = ppr_parts(c, g, a);
  if (e == cudaErrorMemoryAllocation) {
    a.group = 1;
    e = ppr_parts(c, g, a);
  }
  TRY_CUDA_ST(e);
  return PRX_OK;
}

// Teleport entries of columns [c0, c0 + cols) sorted by (vertex, column).
static int ppr_teleport(prx_context* c, uint32_t n, const uint32_t* seed_off, const uint32_t* seeds, uint32_t c0,
                        uint32_t cols, PprArgs& a) {
  PprWs& w = *c->ppr;
  cudaStream_t s = c->stream;
  struct Ent { uint32_t v, col; double m; };
  std::vector<Ent> ent;
  ent.reserve(seed_off[c0 + cols] - seed_off[c0]);
  for (uint32_t k = 0; k < cols; ++k) {
    const uint32_t b = seed_off[c0 + k], e = seed_off[c0 + k + 1];
    const double m = 1.0 / (double)(e - b);
    for (uint32_t i = b; i < e; ++i) ent.push_back({seeds[i], k, m});
  }
  std::sort(ent.begin(), ent.end(), [](const Ent& x, const Ent& y) { return x.v != y.v ? x.v < y.v : x.col < y.col; });
  const size_t ne = ent.size();
  std::vector<uint32_t> hv(ne), hc(ne);
  std::vector<double> hm(ne);
  for (size_t i = 0; i < ne; ++i) {
    hv[i] = ent[i].v;
    hc[i] = ent[i].col;
    hm[i] = ent[i].m;
  }
  TRY_CUDA_ST(grow(&w.tent, w.t_cap, 2 * ne));
  TRY_CUDA_ST(grow(&w.tmass, w.tm_cap, ne));
  TRY_CUDA_ST(cudaMemcpyAsync(w.tent, hv.data(), 4 * ne, cudaMemcpyHostToDevice, s));
  TRY_CUDA_ST(cudaMemcpyAsync(w.tent + ne, hc.data(), 4 * ne, cudaMemcpyHostToDevice, s));
  TRY_CUDA_ST(cudaMemcpyAsync(w.tmass, hm.data(), 8 * ne, cudaMemcpyHostToDevice, s));
  k_ppr_toff<<<grid_for((uint64_t)n + 1, 256, c->sms * 16), 256, 0, s>>>(w.tent, (uint32_t)ne, n, w.toff);
  // the host vectors must outlive the copies
  TRY_CUDA_ST(cudaStreamSynchronize(s));
  a.toff = w.toff;
  a.tcol = w.tent + ne;
  a.tmass = w.tmass;
  return PRX_OK;
}

// Reads the control block back (one sync).
static int ppr_check(prx_context* c) {
  TRY_CUDA_ST(cudaGetLastError());
  TRY_CUDA_ST(cudaMemcpyAsync(&c->st_host[1], c->st, sizeof(State), cudaMemcpyDeviceToHost, c->stream));
  TRY_CUDA_ST(cudaStreamSynchronize(c->stream));
  return PRX_OK;
}

// The iteration loop of one column block as one CUDA graph launch (see the
// file comment); on return st_host[1] holds the control block.  Kernel
// launches inside the graph are counted into *body_launches from the
// control block (FP64 sweeps, FP32 sweeps).
static int ppr_block_graph(prx_context* c, PprArgs& a, const prx_options& o, bool fp32, uint64_t* body_launches) {
  cudaStream_t s = c->stream, s2 = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int st = PRX_OK;
  const int cap = (o.max_iterations < (1 << 30) ? o.max_iterations : (1 << 30)) + 2;
  uint64_t sweep_l = 0, sweep32_l = 0;
  cudaError_t e = cudaGraphCreate(&graph, 0);
  cudaGraphConditionalHandle ho{}, hi{};
  if (e == cudaSuccess) e = cudaGraphConditionalHandleCreate(&ho, graph, 1, cudaGraphCondAssignDefault);
  cudaGraphNodeParams p{};
  p.type = cudaGraphNodeTypeConditional;
  p.conditional.handle = ho;
  p.conditional.type = cudaGraphCondTypeWhile;
  p.conditional.size = 1;
  cudaGraphNode_t node;
  if (e == cudaSuccess) e = cudaGraphAddNode(&node, graph, nullptr, nullptr, 0, &p);
  if (e == cudaSuccess && fp32) e = cudaStreamCreateWithFlags(&s2, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaStreamBeginCaptureToGraph(s, p.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                                          cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    cudaError_t ec = cudaSuccess;
    if (!fp32) {
      ppr_sweep<PPR_J64>(a, c->sms, s, sweep_l);
      k_ppr_fin64<<<1, 1, 0, s>>>(a.st);
      k_ppr_cond<<<1, 1, 0, s>>>(ho, a.st, cap, 0);
    } else {
      // the inner handle belongs to the outer body, the graph being captured
      cudaStreamCaptureStatus cs;
      cudaGraph_t body = nullptr;
      const cudaGraphNode_t* deps = nullptr;
      const cudaGraphEdgeData* edata = nullptr;
      size_t ndeps = 0;
      ec = cudaStreamGetCaptureInfo(s, &cs, nullptr, &body, nullptr, nullptr, nullptr);
      if (ec == cudaSuccess) ec = cudaGraphConditionalHandleCreate(&hi, body, 0, 0);
      if (ec == cudaSuccess) {
        ppr_sweep<PPR_R64>(a, c->sms, s, sweep_l);
        k_ppr_fin_r64<<<1, 1, 0, s>>>(a.st);
        k_ppr_arm_inner<<<1, 1, 0, s>>>(hi, a.st);
        ec = cudaStreamGetCaptureInfo(s, &cs, nullptr, &body, &deps, &edata, &ndeps);
      }
      cudaGraphNodeParams pi{};
      pi.type = cudaGraphNodeTypeConditional;
      pi.conditional.handle = hi;
      pi.conditional.type = cudaGraphCondTypeWhile;
      pi.conditional.size = 1;
      cudaGraphNode_t inode;
      if (ec == cudaSuccess) ec = cudaGraphAddNode(&inode, body, deps, edata, ndeps, &pi);
      if (ec == cudaSuccess) ec = cudaStreamUpdateCaptureDependencies(s, &inode, nullptr, 1,
                                                                      cudaStreamSetCaptureDependencies);
      // the FP32 sweeps of a round: the inner body, captured on a second stream
      if (ec == cudaSuccess) ec = cudaStreamBeginCaptureToGraph(s2, pi.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                                                cudaStreamCaptureModeThreadLocal);
      if (ec == cudaSuccess) {
        ppr_sweep<PPR_S32>(a, c->sms, s2, sweep32_l);
        k_ppr_fin32<<<1, 1, 0, s2>>>(a.st);
        k_ppr_cond_inner<<<1, 1, 0, s2>>>(hi, a.st, cap);
        const cudaError_t el = cudaGetLastError();
        cudaGraph_t inner = nullptr;
        ec = cudaStreamEndCapture(s2, &inner);
        if (ec == cudaSuccess) ec = el;
      }
      if (ec == cudaSuccess) {
        k_ppr_commit<<<grid_for((size_t)a.n * a.cols, 256, c->sms * 16), 256, 0, s>>>(a);
        k_ppr_cond<<<1, 1, 0, s>>>(ho, a.st, cap, 1);
      }
    }
    const cudaError_t el = cudaGetLastError();
    cudaGraph_t captured = nullptr;
    e = cudaStreamEndCapture(s, &captured);  // always leave capture mode
    if (e == cudaSuccess) e = ec;
    if (e == cudaSuccess) e = el;
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
  if (e == cudaSuccess) e = cudaGraphLaunch(exec, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&c->st_host[1], c->st, sizeof(State), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    set_error(std::string("prx_solve_ppr_batched (graph loop): ") + cudaGetErrorString(e));
    st = e == cudaErrorMemoryAllocation ? PRX_ENOMEM : PRX_ECUDA;
  }
  if (exec) cudaGraphExecDestroy(exec);
  if (graph) cudaGraphDestroy(graph);
  if (s2) cudaStreamDestroy(s2);
  if (!st) {
    const State& h = c->st_host[1];
    if (!fp32) {
      *body_launches = (uint64_t)h.iter * (sweep_l + 2);
    } else {
      const uint64_t n64 = (uint64_t)h.rounds, n32 = (uint64_t)(h.iter - h.rounds);
      *body_launches = n64 * (sweep_l + 5) + n32 * (sweep32_l + 2);
    }
  }
  return st;
}

// One column block; the answer's FP64 rows are left in *answer.
static int ppr_block(prx_context* c, const GraphDev& g, PprArgs& a, const prx_options& o, bool fp32,
                     const double** answer, prx_ppr_result* res) {
  cudaStream_t s = c->stream;
  uint64_t& L = c->launches;
  const size_t rows = (size_t)g.n * a.cols;
  TRY_CUDA_ST(cudaMemsetAsync(a.x[0], 0, sizeof(double) * rows, s));
  k_ppr_init<<<grid_for(g.n, 256, c->sms * 16), 256, 0, s>>>(a);
  launch_state_reset(c->st, o.max_iterations, o.tolerance, s);
  L += 2;
  int st;
  if (o.loop != PRX_LOOP_HOST && o.max_iterations > 0) {
    uint64_t body = 0;
    if ((st = ppr_block_graph(c, a, o, fp32, &body))) return st;
    L += body;
    res->graph_launches += 1;
    const State& h = c->st_host[1];
    if (!fp32) {
      *answer = a.x[h.iter & 1];
      res->fp64_sweeps += h.iter;
    } else {
      *answer = h.done ? a.x[1] : a.x[0];  // a converged (or capped) FP64 sweep, else the committed base
      res->fp64_sweeps += h.rounds;
      res->fp32_sweeps += h.iter - h.rounds;
      res->refinements += h.rounds;
    }
    res->iterations = std::max(res->iterations, h.iter);
    res->last_delta = std::max(res->last_delta, h.last_delta);
    return PRX_OK;
  }
  if (!fp32) {
    if (o.max_iterations > 0) {
      for (int k = 1;; k = std::min(2 * k, 16)) {
        for (int i = 0; i < k; ++i) {
          ppr_sweep<PPR_J64>(a, c->sms, s, L);
          k_ppr_fin64<<<1, 1, 0, s>>>(c->st);
          ++L;
        }
        if ((st = ppr_check(c))) return st;
        if (c->st_host[1].done) break;
      }
    } else if ((st = ppr_check(c))) {
      return st;
    }
    const State& h = c->st_host[1];
    *answer = a.x[h.iter & 1];
    res->fp64_sweeps += h.iter;
    res->iterations = std::max(res->iterations, h.iter);
    res->last_delta = std::max(res->last_delta, h.last_delta);
    return PRX_OK;
  }
  int fp64 = 0;
  if (o.max_iterations <= 0) {
    if ((st = ppr_check(c))) return st;
    *answer = a.x[0];
    return PRX_OK;
  }
  for (;;) {
    ppr_sweep<PPR_R64>(a, c->sms, s, L);
    k_ppr_fin_r64<<<1, 1, 0, s>>>(c->st);
    ++L;
    ++fp64;
    if ((st = ppr_check(c))) return st;
    if (c->st_host[1].done) {
      *answer = a.x[1];
      break;
    }
    for (int k = 1;; k = std::min(2 * k, 16)) {
      for (int i = 0; i < k; ++i) {
        ppr_sweep<PPR_S32>(a, c->sms, s, L);
        k_ppr_fin32<<<1, 1, 0, s>>>(c->st);
        ++L;
      }
      if ((st = ppr_check(c))) return st;
      if (c->st_host[1].inner_done) break;
    }
    k_ppr_commit<<<grid_for(rows, 256, c->sms * 16), 256, 0, s>>>(a);
    ++L;
    if (c->st_host[1].iter >= o.max_iterations) {
      TRY_CUDA_ST(cudaStreamSynchronize(s));
      *answer = a.x[0];
      break;
    }
  }
  const State& h = c->st_host[1];
  res->fp64_sweeps += fp64;
  res->fp32_sweeps += h.iter - fp64;
  res->refinements += h.rounds;
  res->iterations = std::max(res->iterations, h.iter);
  res->last_delta = std::max(res->last_delta, h.last_delta);
  return PRX_OK;
}

static int ppr_common(prx_context* c, prx_graph* gr, uint32_t nvec, const uint32_t* seed_off, const uint32_t* seeds,
                      const prx_options* opt, double* ranks_out, prx_ppr_result* res, bool device_out) {
  if (!c || !gr || gr->ctx != c) FAIL(PRX_EINVAL, "prx_solve_ppr_batched: bad context or graph");
  if (nvec == 0 || !seed_off || !seeds) FAIL(PRX_EINVAL, "prx_solve_ppr_batched: no teleport vectors");
  prx_options o;
  if (opt) o = *opt;
  else prx_options_default(&o);
  if (o.precision != PRX_FP64 && o.precision != PRX_FP32_REFINE)
    FAIL(PRX_EINVAL, "prx_solve_ppr_batched: unknown precision");
  if (!(o.damping >= 0 && o.damping < 1)) FAIL(PRX_EINVAL, "prx_solve_ppr_batched: damping must be in [0, 1)");
  const GraphDev& g = gr->g;
  if (seed_off[0] != 0) FAIL(PRX_EINVAL, "prx_solve_ppr_batched: seed_off[0] must be 0");
  for (uint32_t k = 0; k < nvec; ++k)
    if (seed_off[k + 1] <= seed_off[k]) FAIL(PRX_EINVAL, "prx_solve_ppr_batched: every seed set must be non-empty");
  for (uint32_t i = 0; i < seed_off[nvec]; ++i)
    if (seeds[i] >= g.n) FAIL(PRX_EINVAL, "prx_solve_ppr_batched: seed id out of range");
  prx_ppr_result r{};
  if (g.n == 0) {
    if (res) *res = r;
    return PRX_OK;
  }
  if (!ranks_out) FAIL(PRX_EINVAL, "prx_solve_ppr_batched: ranks_out is NULL");
  TRY_CUDA_ST(cudaSetDevice(c->device));
  const bool fp32 = o.precision == PRX_FP32_REFINE;
  int st = ppr_ws(c, g.n, fp32);
  if (st) return st;
  PprWs& w = *c->ppr;
  cudaStream_t s = c->stream;
  PoolBlock pairs{s};  // PprArgs::pair
  PprArgs a{};
  a.xtoff = g.xtoff;
  a.xtbase = g.xtbase;
  a.seg_shift = g.seg_shift;
  a.rcp = g.rcp;
  a.rcp32 = g.rcp32;
  a.xtedg = g.xtedg;
  a.x[0] = w.x[0];
  a.x[1] = w.x[1];
  a.rho = w.rho;
  a.e[0] = w.e[0];
  a.e[1] = w.e[1];
  a.st = c->st;
  a.n = g.n;
  a.P = o.damping;
  a.Q = 1.0 - o.damping;
  a.P32 = (float)o.damping;
  a.low_max = g.ppr_low_max ? g.ppr_low_max : kLowMax;
  a.seg = g.ppr_seg ? g.ppr_seg : kSeg;
  r.low_max = a.low_max;
  r.seg_edges = a.seg;
  a.per = a.seg / kSegParts;
  if ((st = ppr_segments(c, g, a))) return st;
  double* out = ranks_out;
  const size_t total = (size_t)g.n * nvec;
  if (!device_out) {
    TRY_CUDA_ST(grow(&w.out, w.out_cap, total));
    out = w.out;
  }
  const uint64_t l0 = c->launches;
  TRY_CUDA_ST(cudaEventRecord(c->ev[0], s));
  // The LOW rows in order of length (rows side by side in a warp then end
  // together); by id with another bound, with row segments, or without memory
  // for the list.
  bool by_length = a.low_max == kLowMax && g.nseg == 1;
  if (by_length) {
    const cudaError_t e = ensure_len_list(gr->g, c->sms, s);
    if (e != cudaErrorMemoryAllocation) TRY_CUDA_ST(e);
    by_length = e == cudaSuccess;
  }
  a.rows = by_length ? g.len_list : nullptr;
  a.nrows = by_length ? g.cls_begin[MID] : g.n;
  a.flat = !mixed_lengths(g);
  if (fp32 && (!a.flat || a.nparts || (nvec % kCols && nvec % kCols <= 48))) {  // not k_ppr_flat alone
    const uint64_t slots = g.nseg > 1 ? g.xtpos.back() + (g.m - g.xtseg0.back()) : g.m;
    const cudaError_t e = graph_alloc(&pairs.p, sizeof(uint2) * slots, s);
    if (e != cudaErrorMemoryAllocation) TRY_CUDA_ST(e);
    if (e == cudaSuccess) {
      uint2* pair = static_cast<uint2*>(pairs.p);
      k_ppr_pairs<<<grid_for(slots, 256, c->sms * 32), 256, 0, s>>>(g.xtedg, slots, g.n, g.rcp32, pair);
      c->launches += 1;
      a.pair = pair;
    }
  }
  for (uint32_t c0 = 0; c0 < nvec; c0 += kCols) {
    const uint32_t cols = std::min<uint32_t>(kCols, nvec - c0);
    for (int w : {64, 48, 32, 24, 16, 8})
      if ((int)cols <= w) a.cols = w;
    if ((st = ppr_teleport(c, g.n, seed_off, seeds, c0, cols, a))) return st;
    const double* answer = nullptr;
    if ((st = ppr_block(c, g, a, o, fp32, &answer, &r))) return st;
    k_ppr_out<<<grid_for((uint64_t)g.n * cols, 256, c->sms * 16), 256, 0, s>>>(answer, g.n, (uint32_t)a.cols, nvec, c0, cols, out);
    c->launches += 1;
  }
  TRY_CUDA_ST(cudaEventRecord(c->ev[1], s));
  if (!device_out) TRY_CUDA_ST(cudaMemcpyAsync(ranks_out, out, sizeof(double) * total, cudaMemcpyDeviceToHost, s));
  TRY_CUDA_ST(cudaStreamSynchronize(s));
  TRY_CUDA_ST(cudaGetLastError());
  float ms = 0;
  TRY_CUDA_ST(cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]));
  r.time_ms = ms;
  r.kernel_launches = c->launches - l0;
  if (res) *res = r;
  return PRX_OK;
}

extern "C" {

int prx_solve_ppr_batched(prx_context* c, prx_graph* gr, uint32_t nvec, const uint32_t* seed_off,
                          const uint32_t* seeds, const prx_options* o, double* ranks_out, prx_ppr_result* res) {
  return ppr_common(c, gr, nvec, seed_off, seeds, o, ranks_out, res, false);
}

int prx_solve_ppr_batched_device(prx_context* c, prx_graph* gr, uint32_t nvec, const uint32_t* seed_off,
                                 const uint32_t* seeds, const prx_options* o, double* ranks_out,
                                 prx_ppr_result* res) {
  return ppr_common(c, gr, nvec, seed_off, seeds, o, ranks_out, res, true);
}

// Times short FP32-refined solves (64 teleport vectors of one seed each, 1
// FP64 and 5 FP32 sweeps, best of two) over the warp-per-vertex bound
// (64, 256, 1024) and the segment width (256, 512, 1024, 2048 in-edges), and
// keeps the fastest pair on the graph for its later solves.
int prx_autotune_ppr(prx_context* c, prx_graph* gr, prx_ppr_tune_result* out) {
  if (!c || !gr || gr->ctx != c) FAIL(PRX_EINVAL, "prx_autotune_ppr: bad context or graph");
  GraphDev& g = gr->g;
  prx_ppr_tune_result best{};
  if (g.n == 0) {
    if (out) *out = best;
    return PRX_OK;
  }
  TRY_CUDA_ST(cudaSetDevice(c->device));
  const uint32_t nvec = kCols;
  std::vector<uint32_t> off(nvec + 1), seeds(nvec);
  for (uint32_t k = 0; k < nvec; ++k) {
    off[k] = k;
    seeds[k] = (uint32_t)((uint64_t)k * g.n / nvec);
  }
  off[nvec] = nvec;
  double* ranks = nullptr;
  TRY_CUDA_ST(device_alloc(&ranks, sizeof(double) * (size_t)g.n * nvec));
  prx_options o;
  prx_options_default(&o);
  o.precision = PRX_FP32_REFINE;
  o.tolerance = 0.0;
  o.max_iterations = 6;
  const uint32_t lows[] = {64, 256, 1024}, segs[] = {256, 512, 1024, 2048};
  const uint32_t keep_low = g.ppr_low_max, keep_seg = g.ppr_seg;
  float best_ms = 0;
  int trials = 0, st = PRX_OK;
  for (uint32_t lo : lows) {
    for (uint32_t sg : segs) {
      g.ppr_low_max = lo;
      g.ppr_seg = sg;
      float ms = 0;
      for (int rep = 0; rep < 2 && !st; ++rep) {
        prx_ppr_result r{};
        st = ppr_common(c, gr, nvec, off.data(), seeds.data(), &o, ranks, &r, true);
        if (!st && (rep == 0 || r.time_ms < ms)) ms = r.time_ms;
      }
      if (st) break;
      ++trials;
      if (!best.trials || ms < best_ms) {
        best_ms = ms;
        best.low_max = lo;
        best.seg_edges = sg;
        best.trials = 1;
      }
    }
    if (st) break;
  }
  cudaFree(ranks);
  if (st) {
    g.ppr_low_max = keep_low;
    g.ppr_seg = keep_seg;
    return st;
  }
  g.ppr_low_max = best.low_max;
  g.ppr_seg = best.seg_edges;
  best.ms_per_solve = best_ms;
  best.trials = trials;
  if (out) *out = best;
  return PRX_OK;
}

}  // extern "C"
