// prx_weighted.cu -- weighted PageRank and its adjoint.  No counterpart in
// the reference, whose graphs are unweighted (xtdat holds integer
// out-degrees, inc/pagerankCuda.hxx:87-109).
//
// Edge u -> v carries a weight w_uv > 0; rows are normalised,
// P_uv = w_uv / W_u with W_u = sum_v w_uv, and
//   forward:  r = (1 - alpha) t + alpha P^T r         (pull over in-edges)
//   adjoint:  lambda = alpha P lambda + g             (pull over out-edges)
// where g = dL/dr.  Both are Jacobi iterations of one pull kernel family,
// run on the in-CSR (forward) or on the out-CSR (adjoint, the reversed
// graph), stopped by the reference's L-inf test (:680,689).  With lambda and
// the converged r:
//   dL/dw_uv   = (r_u / W_u) (alpha lambda_v - lambda_u + g_u)
//   dL/dt      = (1 - alpha) lambda
//   dL/dalpha  = lambda . (P^T r - t)
// (dr = (I - alpha P^T)^-1 (alpha dP^T r + (P^T r - t) dalpha + (1-alpha) dt),
// and dP_uv'/dw_uv = (delta_vv' - P_uv') / W_u.)
//
// Rows go by length class: <= 64 one thread per row, then one warp, then one
// block; every sum has a fixed order, so results are deterministic.  Graphs
// up to the lines of persist_fits iterate in one cooperative kernel
// (k_pull_persist), as the FP64 solves do (prx_persist.cu): a sweep of R-MAT
// 2^18 (4.2M edges, everything in L2) took 83 us in four launches and takes
// 24 us there.  Larger ones launch the classes one by one.
//
// Graphs with row segments (64-bit offsets, see GraphDev): px / pt are laid
// out like the edge arrays they follow (the same segment bases), and the
// weights and dL/dw stay in the compact out-CSR order a caller uses (edge j
// of a segment at its compact start + j).
#include <algorithm>
#include "prx_ctx.h"
#include "prx_update.cuh"

namespace prx {

void drop_weights(GraphDev& g) {
  cudaFree(g.px);
  cudaFree(g.pt);
  cudaFree(g.wsum);
  cudaFree(g.wseg);
  cudaFree(g.tpos);
  g.px = g.pt = g.wsum = nullptr;
  g.wseg = nullptr;
  g.tpos = nullptr;
  g.tpos_built = g.weights_set = false;
}

struct PullArgs {
  const uint32_t* off;            // rows to pull over
  const uint32_t* edg;
  const double* prob;             // P of each edge of the rows (laid out like edg)
  const unsigned long long* seg;  // row segments: the bases of edg and prob (null: one segment)
  uint32_t shift;
  const uint32_t* list;           // row ids by class
  uint32_t begin[NCLS + 1];
  const double* base;             // b_v, or base_const when null
  double base_scale;              // y_v = base_scale * b_v + alpha * sum
  double base_const;
  double alpha;
  const double* xin;              // null: the iterate of parity st->iter & 1
  double* x[2];
  double* y;                      // single sweep output (xin set)
  State* st;                      // null: single sweep, no L-inf
  uint32_t n;
  // the persistent loop's rows (null: not taken)
  const uint32_t* plan;
  const uint32_t* plan_low;
  uint32_t plan_begin[NCLS + 1];
  bool solo;
};

__device__ __forceinline__ const double* pull_src(const PullArgs& a) {
  return a.xin ? a.xin : a.x[a.st->iter & 1];
}

__device__ __forceinline__ unsigned long long pull_finish(const PullArgs& a, uint32_t v, double sum) {
  const double b = a.base ? a.base[v] : a.base_const;
  const double y = fma(a.alpha, sum, a.base_scale * b);
  if (!a.st) {
    a.y[v] = y;
    return 0;
  }
  const int p = a.st->iter & 1;
  const double old = a.x[p][v];
  a.x[p ^ 1][v] = y;
  return dbits(fabs(y - old));
}

__global__ void __launch_bounds__(256) k_pull_low(PullArgs a) {
  if (a.st && a.st->done) return;
  const double* __restrict__ x = pull_src(a);
  unsigned long long emax = 0;
  for (uint32_t i = a.begin[LOW] + blockIdx.x * blockDim.x + threadIdx.x; i < a.begin[MID];
       i += gridDim.x * blockDim.x) {
    const uint32_t v = a.list[i];
    const uint64_t iv = seg_index(v, a.shift);
    const uint32_t s = a.off[iv], e = a.off[iv + 1];
    const uint64_t b = a.seg ? a.seg[(uint64_t)v >> a.shift] : 0;
    const uint32_t* __restrict__ edg = a.edg + b;
    const double* __restrict__ prob = a.prob + b;
    double acc = 0.0;
    uint32_t j = s;
    for (; j + 2 <= e; j += 2) {
      const uint32_t u0 = __ldg(edg + j), u1 = __ldg(edg + j + 1);
      const double p0 = __ldg(prob + j), p1 = __ldg(prob + j + 1);
      const double x0 = __ldg(x + u0), x1 = __ldg(x + u1);
      acc = fma(p0, x0, acc);
      acc = fma(p1, x1, acc);
    }
    if (j < e) acc = fma(__ldg(prob + j), __ldg(x + __ldg(edg + j)), acc);
    const unsigned long long d = pull_finish(a, v, acc);
    emax = d > emax ? d : emax;
  }
  if (a.st) block_max_bits(emax, &a.st->el_bits[a.st->iter & 1]);
}

__global__ void __launch_bounds__(256) k_pull_mid(PullArgs a) {
  if (a.st && a.st->done) return;
  const double* __restrict__ x = pull_src(a);
  const uint32_t lane = lane_id();
  unsigned long long emax = 0;
  for (uint32_t i = a.begin[MID] + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < a.begin[HIGH];
       i += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t v = a.list[i];
    const uint64_t iv = seg_index(v, a.shift);
    const uint32_t s = a.off[iv], e = a.off[iv + 1];
    const uint64_t b = a.seg ? a.seg[(uint64_t)v >> a.shift] : 0;
    const uint32_t* __restrict__ edg = a.edg + b;
    const double* __restrict__ prob = a.prob + b;
    double acc = 0.0;
    for (uint32_t j = s + lane; j < e; j += 32) acc = fma(__ldg(prob + j), __ldg(x + __ldg(edg + j)), acc);
#pragma unroll
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
      const unsigned long long d = pull_finish(a, v, acc);
      emax = d > emax ? d : emax;
    }
  }
  if (a.st) block_max_bits(emax, &a.st->el_bits[a.st->iter & 1]);
}

__global__ void __launch_bounds__(256) k_pull_high(PullArgs a) {
  __shared__ double part[8];
  if (a.st && a.st->done) return;
  const double* __restrict__ x = pull_src(a);
  unsigned long long emax = 0;
  for (uint32_t i = a.begin[HIGH] + blockIdx.x; i < a.begin[NCLS]; i += gridDim.x) {
    const uint32_t v = a.list[i];
    const uint64_t iv = seg_index(v, a.shift);
    const uint32_t s = a.off[iv], e = a.off[iv + 1];
    const uint64_t b = a.seg ? a.seg[(uint64_t)v >> a.shift] : 0;
    const uint32_t* __restrict__ edg = a.edg + b;
    const double* __restrict__ prob = a.prob + b;
    double acc = 0.0;
    for (uint32_t j = s + threadIdx.x; j < e; j += 256) acc = fma(__ldg(prob + j), __ldg(x + __ldg(edg + j)), acc);
#pragma unroll
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane_id() == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int k = 0; k < 8; ++k) t += part[k];
      const unsigned long long d = pull_finish(a, v, t);
      emax = d > emax ? d : emax;
    }
    __syncthreads();
  }
  if (a.st) block_max_bits(emax, &a.st->el_bits[a.st->iter & 1]);
}

__global__ void k_pull_fin(State* st) {
  if (st->done) return;
  const int p = st->iter & 1;
  const double el = __longlong_as_double((long long)st->el_bits[p]);
  st->last_delta = el;
  st->iter += 1;
  st->el_bits[p ^ 1] = 0;
  if (el < st->tol || st->iter >= st->max_iter) st->done = 1;
}

// ---- the loop as one cooperative kernel ------------------------------------
// Rows of PullArgs::list by class with kPlanMid as the MID / HIGH boundary.
// See prx_persist.cu for the split, the memory rules and the barrier; the
// iterate is read by ordinary loads.
struct PullRow {
  uint32_t v, len;
  uint64_t at;   // the row's first edge in edg and prob
};
__device__ __forceinline__ PullRow pull_row(const PullArgs& a, uint32_t v) {
  const uint64_t iv = seg_index(v, a.shift);
  const uint32_t s = __ldg(a.off + iv);
  return {v, __ldg(a.off + iv + 1) - s, (a.seg ? a.seg[(uint64_t)v >> a.shift] : 0) + s};
}

__global__ void __launch_bounds__(256, 3) k_pull_persist(PullArgs a, const uint32_t* __restrict__ low) {
  __shared__ double part[8];
  __shared__ double s_tree[8][RowTree::kSlots];
  __shared__ unsigned long long s_el;
  State* st = a.st;
  if (st->done) return;
  const uint32_t lane = lane_id(), t = threadIdx.x;
  const RowTree tree{s_tree[t >> 5]};
  const WarpShare share(a.begin[NCLS] - a.begin[HIGH], a.solo);
  const uint32_t warps = share.warps, warp = share.warp;
  const uint32_t nlow = a.begin[MID] - a.begin[LOW], nmid = a.begin[HIGH] - a.begin[MID];
  const uint32_t units = nmid + (nlow + 31) / 32;
  const uint32_t low0 = warp < nmid ? warp + (nmid - warp + warps - 1) / warps * warps : warp;
  // unit u: a MID row in every lane, or a LOW row per lane (len 0: none)
  auto load_unit = [&](uint32_t u) -> PullRow {
    if (u < nmid) return pull_row(a, __ldg(a.list + a.begin[MID] + u));
    const uint32_t i = 32 * (u - nmid) + lane;
    return i < nlow ? pull_row(a, __ldg(low + i)) : PullRow{0, 0, 0};
  };
  PullRow coming{0, 0, 0};  // loaded while the unit before is summed
  if (warp < units) coming = load_unit(warp);
  auto take = [&](uint32_t u) {
    const PullRow r = coming;
    if (units > warps) coming = load_unit(u + warps < units ? u + warps : warp);
    return r;
  };
  const int max_iter = st->max_iter;
  const double tol = st->tol;
  GridBarrier bar(st);
  for (int it = 0;; ++it) {
    const int p = it & 1;
    const double* x = a.x[p];
    unsigned long long emax = 0;
    auto finish = [&](uint32_t v, double sum, double old, double b) {
      const double y = fma(a.alpha, sum, b);
      a.x[p ^ 1][v] = y;
      const unsigned long long d = dbits(fabs(y - old));
      emax = d > emax ? d : emax;
    };
    auto base = [&](uint32_t v) { return a.base_scale * (a.base ? __ldg(a.base + v) : a.base_const); };
    // sum of a row's terms i0, i0 + step, ... below len (steps: as many as any
    // lane has; an FP64 fma issued for no term costs as much as one): ids and
    // probabilities of the next four are loaded behind the gathers of these
    auto strided = [&](const PullRow& r, uint32_t i0, uint32_t step, uint32_t steps) {
      const uint32_t* __restrict__ edg = a.edg + r.at;
      const double* __restrict__ prob = a.prob + r.at;
      uint32_t u[4];
      double w[4];
      auto load = [&](uint32_t j) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t i = j + k * step;
          u[k] = i < r.len ? __ldg(edg + i) : 0u;
          w[k] = i < r.len ? __ldg(prob + i) : 0.0;
        }
      };
      double acc = 0.0;
      load(i0);
      for (uint32_t n = steps, j = i0; n; j += 4 * step) {
        double g[4], q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          g[k] = j + k * step < r.len ? x[u[k]] : 0.0;
          q[k] = w[k];
        }
        load(j + 4 * step);
        if (n >= 4) {
#pragma unroll
          for (int k = 0; k < 4; ++k) acc = fma(q[k], g[k], acc);
          n -= 4;
        } else {  // lanes past their row add 0 * 0
          switch (n) {
            case 1: acc = fma(q[0], g[0], acc); break;
            case 2: acc = fma(q[1], g[1], fma(q[0], g[0], acc)); break;
            default: acc = fma(q[2], g[2], fma(q[1], g[1], fma(q[0], g[0], acc))); break;
          }
          n = 0;
        }
      }
      return acc;
    };
    for (uint32_t i = a.begin[HIGH] + share.row; i < a.begin[NCLS]; i += gridDim.x) {
      const PullRow r = pull_row(a, __ldg(a.list + i));
      double acc = strided(r, t, 256, (r.len + 255) / 256);
#pragma unroll
      for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) part[t >> 5] = acc;
      __syncthreads();
      if (t == 0) {
        double sum = 0.0;
        for (int k = 0; k < 8; ++k) sum += part[k];
        finish(r.v, sum, x[r.v], base(r.v));
      }
      __syncthreads();
    }
    // four MID rows are folded and finished together (see RowTree)
    uint32_t qv = 0, held = 0;
    double qold = 0.0, qb = 0.0;
    auto flush = [&] {
      double z = tree.fold<false>(held);
      z = __shfl_sync(0xffffffffu, z, (lane & 3u) * 8);
      if (lane < held) finish(qv, z, qold, qb);
      held = 0;
    };
    for (uint32_t u = warp; u < nmid; u += warps) {
      const PullRow r = take(u);
      if (lane == held) {
        qv = r.v;
        qold = x[r.v];
        qb = base(r.v);
      }
      tree.put(held++, strided(r, lane, 32, (r.len + 31) / 32));
      if (held == RowTree::kRows) flush();
    }
    if (held) flush();
    for (uint32_t u = low0; u < units; u += warps) {
      const PullRow r = take(u);
      const bool mine = 32 * (u - nmid) + lane < nlow;
      const double old = mine ? x[r.v] : 0.0, b = mine ? base(r.v) : 0.0;
      const double sum = strided(r, 0, 1, __reduce_max_sync(0xffffffffu, r.len));
      if (mine) finish(r.v, sum, old, b);
    }
    block_max_bits(emax, &st->pel[it % 3]);
    if (blockIdx.x == 0 && t == 0) st->pel[(it + 1) % 3] = 0;
    if (!bar.sync([&] { s_el = *(volatile unsigned long long*)&st->pel[it % 3]; })) return;
    const double el = __longlong_as_double((long long)s_el);
    if (el < tol || it + 1 >= max_iter) {
      if (blockIdx.x == 0 && t == 0) {
        st->iter = it + 1;
        st->last_delta = el;
        st->done = 1;
      }
      return;
    }
  }
}

static int pull_grid(uint64_t work, int per_block, int cap) {
  const uint64_t b = (work + per_block - 1) / per_block;
  return (int)std::max<uint64_t>(1, std::min<uint64_t>(b, (uint64_t)cap));
}

static void pull_sweep(const PullArgs& a, int sms, cudaStream_t s, uint64_t& launches) {
  const uint32_t nl = a.begin[MID] - a.begin[LOW], nm = a.begin[HIGH] - a.begin[MID];
  const uint32_t nh = a.begin[NCLS] - a.begin[HIGH];
  if (nl) { k_pull_low<<<pull_grid(nl, 256, sms * 8), 256, 0, s>>>(a); ++launches; }
  if (nm) { k_pull_mid<<<pull_grid(nm, 8, sms * 8), 256, 0, s>>>(a); ++launches; }
  if (nh) { k_pull_high<<<pull_grid(nh, 1, sms * 4), 256, 0, s>>>(a); ++launches; }
}

// ---- weights ---------------------------------------------------------------------
// Warp per source u: W_u (lane-strided partial sums folded in lane order), px,
// and each out-edge's probability scattered to its in-CSR slot (binary search
// of u in v's ascending in-row).  err: 1 bad weight, 2 edge missing in xt.
// (Graph addressing of both CSRs: see the file comment; wseg: each out-CSR
// segment's compact start, null for one segment.)
struct WeightCsr {
  const uint32_t *xoff, *xedg, *xtoff, *xtedg;
  const unsigned long long *xbase, *xtbase, *wseg;
  uint32_t shift;
  uint32_t* tpos;   // GraphDev::tpos (null: no memory for it, every call searches)
};

// p = w / W_u of an out-edge to its places in px and pt; its position among
// v's in-edges is found once per graph version (tpos, found set).
__device__ __forceinline__ void put_weight(const WeightCsr& c, uint32_t u, uint64_t at, double p, bool found,
                                           double* __restrict__ px, double* __restrict__ pt, uint32_t* err) {
  px[at] = p;
  const uint32_t v = c.xedg[at];
  const uint64_t bv = c.xtbase ? c.xtbase[(uint64_t)v >> c.shift] : 0;
  if (found) {
    pt[bv + c.tpos[at]] = p;
    return;
  }
  const uint64_t iv = seg_index(v, c.shift);
  const uint32_t* row = c.xtedg + bv;
  uint32_t lo = c.xtoff[iv], hi = c.xtoff[iv + 1];
  const uint32_t end = hi;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (row[mid] < u) lo = mid + 1;
    else hi = mid;
  }
  if (lo < end && row[lo] == u) {
    pt[bv + lo] = p;
    if (c.tpos) c.tpos[at] = lo;
  } else {
    atomicOr(err, 2u);
  }
}

// A float as a double by integer operations (the conversion instruction runs
// on the FP64 pipe); zeros, subnormals, infinities and NaN convert as usual.
__device__ __forceinline__ double widen(float x) {
  const uint32_t b = __float_as_uint(x), e = (b >> 23) & 0xffu;
  if (e - 1u >= 254u) return (double)x;
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20))), (int)(b << 29));
}

// w / W correctly rounded from y = RN(1 / W), as div_count does (normal W).
__device__ __forceinline__ double div_by(double w, double W, double y) {
  const double q = w * y;
  return fma(fma(-q, W, w), y, q);
}

__device__ __forceinline__ double checked_weight(float x, uint32_t* err) {
  if (!(x > 0.f) || !(x < INFINITY)) atomicOr(err, 1u);
  return widen(x);
}

// What bounds setting weights: the FP64 pipe.  A warp per row and a plain
// division per edge took 0.28 ms of it on R-MAT 2^18 (rows of 16 edges on
// average), and one hub's row kept its warp busy for 2.5 ms.  Now rows of up
// to 64 edges go by thread (in order of length where they mix), the next ones
// by warp, longer ones by block (k_weight_sums, k_weight_edges), with one
// reciprocal per row and three FP64 operations per edge.  L lanes take a row of up
// to 64: eight where they are four edges long and more (a lane alone reads its row
// piece by piece: 31M edges in even rows of 30 5.1 ms, R-MAT 2^18 0.29; by eight
// 1.29 and 0.18), one for shorter ones (rows of 3 0.09 | 0.26) and for rows of
// mixed lengths past L2 (R-MAT 2^20 0.70 | 0.78).
constexpr uint32_t kSideMixed = 1u << 19;
struct WeightRows {
  const uint32_t *low, *mid;
  uint32_t nlow, nmid;
};

template <uint32_t L>
__global__ void __launch_bounds__(256) k_set_weights(WeightCsr c, WeightRows rows, const float* __restrict__ w,
                                                     bool found, double* __restrict__ wsum, double* __restrict__ px,
                                                     double* __restrict__ pt, uint32_t* err) {
  const uint32_t lane = lane_id(), warps = (gridDim.x * blockDim.x) >> 5;
  constexpr uint32_t G = 32 / L;  // LOW rows side by side
  const uint32_t units = rows.nmid + (rows.nlow + G - 1) / G;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < units; i += warps) {
    const bool mid = i < rows.nmid;
    const uint32_t at = mid ? i : G * (i - rows.nmid) + lane / L;
    const bool row = mid || at < rows.nlow;
    const uint32_t u = row ? (mid ? rows.mid : rows.low)[at] : 0u, first = mid ? lane : lane % L, step = mid ? 32 : L;
    const uint64_t iu = seg_index(u, c.shift);
    const uint32_t s = row ? c.xoff[iu] : 0u, e = row ? c.xoff[iu + 1] : 0u;
    const uint64_t bu = c.xbase ? c.xbase[(uint64_t)u >> c.shift] : 0;  // device position of the row's segment
    const uint64_t wu = c.wseg ? c.wseg[(uint64_t)u >> c.shift] : 0;    // its compact position
    double acc = 0.0;
    for (uint32_t j = s + first; j < e; j += step) acc += checked_weight(w[wu + j], err);
    if (mid) {
#pragma unroll
      for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    } else {
#pragma unroll
      for (int o = L / 2; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    }
    if (row && first == 0) wsum[u] = acc;
    const double y = 1.0 / acc;
    for (uint32_t j = s + first; j < e; j += step)
      put_weight(c, u, bu + j, div_by(widen(w[wu + j]), acc, y), found, px, pt, err);
  }
}

// W_u of the long rows, a block each (256 strided sums, then in order).
__global__ void __launch_bounds__(256) k_weight_sums(WeightCsr c, const float* __restrict__ w,
                                                     const uint32_t* __restrict__ list, double* __restrict__ wsum,
                                                     uint32_t* err) {
  __shared__ double part[8];
  const uint32_t u = list[blockIdx.x];
  const uint64_t iu = seg_index(u, c.shift);
  const uint32_t s = c.xoff[iu], e = c.xoff[iu + 1];
  const uint64_t wu = c.wseg ? c.wseg[(uint64_t)u >> c.shift] : 0;
  double acc = 0.0;
  for (uint32_t j = s + threadIdx.x; j < e; j += 256) {
    acc += checked_weight(w[wu + j], err);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane_id() == 0) part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < 8; ++k) t += part[k];
    wsum[u] = t;
  }
}

// The long rows' edges: block (x, y) takes every gridDim.y-th piece of row x.
__global__ void __launch_bounds__(256) k_weight_edges(WeightCsr c, const float* __restrict__ w,
                                                      const uint32_t* __restrict__ list, bool found,
                                                      const double* __restrict__ wsum, double* __restrict__ px,
                                                      double* __restrict__ pt, uint32_t* err) {
  const uint32_t u = list[blockIdx.x];
  const uint64_t iu = seg_index(u, c.shift);
  const uint32_t s = c.xoff[iu], e = c.xoff[iu + 1];
  const uint64_t bu = c.xbase ? c.xbase[(uint64_t)u >> c.shift] : 0;
  const uint64_t wu = c.wseg ? c.wseg[(uint64_t)u >> c.shift] : 0;
  const double W = wsum[u], y = 1.0 / W;
  for (uint32_t j = s + blockIdx.y * 256 + threadIdx.x; j < e; j += gridDim.y * 256)
    put_weight(c, u, bu + j, div_by(widen(w[wu + j]), W, y), found, px, pt, err);
}

// ---- gradients -------------------------------------------------------------------
// dL/dw_uv = (r_u / W_u) (alpha lambda_v - lambda_u + g_u): a warp per source
// of up to mid_max edges, the pieces of the longer rows (list) by block as in
// k_weight_edges.
__device__ __forceinline__ void grad_row(const WeightCsr& cs, uint32_t u, uint32_t first, uint32_t step,
                                         const double* __restrict__ wsum, const double* __restrict__ r,
                                         const double* __restrict__ lam, const double* __restrict__ g, double alpha,
                                         double* __restrict__ out) {
  const double f = r[u] / wsum[u], c = g[u] - lam[u];
  const uint64_t iu = seg_index(u, cs.shift);
  const uint64_t bu = cs.xbase ? cs.xbase[(uint64_t)u >> cs.shift] : 0;
  const uint64_t wu = cs.wseg ? cs.wseg[(uint64_t)u >> cs.shift] : 0;
  const uint32_t e = cs.xoff[iu + 1];
  for (uint32_t j = cs.xoff[iu] + first; j < e; j += step) out[wu + j] = f * fma(alpha, lam[cs.xedg[bu + j]], c);
}
__global__ void __launch_bounds__(256) k_grad_w(WeightCsr cs, const double* __restrict__ wsum,
                                                const double* __restrict__ r, const double* __restrict__ lam,
                                                const double* __restrict__ g, double alpha, uint32_t n,
                                                uint32_t mid_max, double* __restrict__ out) {
  for (uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n; u += (gridDim.x * blockDim.x) >> 5)
    if (row_len(cs.xoff, cs.shift, u) <= mid_max) grad_row(cs, u, lane_id(), 32, wsum, r, lam, g, alpha, out);
}
__global__ void __launch_bounds__(256) k_grad_w_long(WeightCsr cs, const uint32_t* __restrict__ list,
                                                     const double* __restrict__ wsum, const double* __restrict__ r,
                                                     const double* __restrict__ lam, const double* __restrict__ g,
                                                     double alpha, double* __restrict__ out) {
  grad_row(cs, list[blockIdx.x], blockIdx.y * 256 + threadIdx.x, gridDim.y * 256, wsum, r, lam, g, alpha, out);
}

__global__ void k_fill(double* __restrict__ x, double value, uint32_t n) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) x[v] = value;
}

__global__ void k_scale(const double* __restrict__ x, double f, uint32_t n, double* __restrict__ out) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) out[v] = f * x[v];
}

// Fixed-order dot product lambda . (y - t): per-block partial sums (grid-stride
// order, then the block tree), then one thread adds the partials in order.
__global__ void __launch_bounds__(256) k_dot_part(const double* __restrict__ lam, const double* __restrict__ y,
                                                  const double* __restrict__ t, double tconst, uint32_t n,
                                                  double* __restrict__ part) {
  __shared__ double sh[256];
  double acc = 0.0;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    acc = fma(lam[v], y[v] - (t ? t[v] : tconst), acc);
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int o = 128; o; o >>= 1) {
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

__global__ void k_dot_final(const double* __restrict__ part, int np, double* __restrict__ out) {
  double acc = 0.0;
  for (int i = 0; i < np; ++i) acc += part[i];
  *out = acc;
}

}  // namespace prx

// ---- host side --------------------------------------------------------------------
static int wk_grow(prx_context* c, size_t doubles) {
  if (c->wk && c->wk_cap >= doubles) return PRX_OK;
  cudaFree(c->wk);
  c->wk = nullptr;
  c->wk_cap = 0;
  TRY_CUDA_ST(device_alloc(&c->wk, sizeof(double) * doubles));
  c->wk_cap = doubles;
  return PRX_OK;
}

static WeightCsr weight_csr(const GraphDev& g) {
  return WeightCsr{g.xoff, g.xedg, g.xtoff, g.xtedg, g.xbase, g.xtbase, g.wseg, g.seg_shift, g.tpos};
}

// Device slots of one CSR's edge array (its segments' positions and counts).
static uint64_t csr_slots(const GraphDev& g, const std::vector<uint64_t>& seg0, const std::vector<uint64_t>& pos) {
  if (g.nseg <= 1) return g.m ? g.m : 1;
  return pos.back() + (g.m - seg0.back()) + 4;
}

// Blocks per long row of k_weight_edges and k_grad_w_long.
constexpr int kLongPieces = 8;

// The out-rows by class that the weights and their gradients go by: oplan_list,
// or ocls_list when there was no memory for it.
// LOW ids, MID ones up to mid_max, then the longer ones in two pieces (of oplan_list
// the first MID rows and the HIGH ones).
struct OutRows {
  const uint32_t *low, *mid, *longs[2];
  uint32_t nlow, nmid, nlong[2];
  uint32_t mid_max;
};
static OutRows out_rows(const GraphDev& g) {
  const uint32_t* list = g.oplan_have ? g.oplan_list : g.ocls_list;
  const uint32_t* begin = g.oplan_have ? g.oplan_begin : g.ocls_begin;
  const uint32_t skip = g.oplan_have ? g.oplan_info.mid_long : 0, nmid = begin[HIGH] - begin[MID];
  return {list, list + begin[MID] + skip, {list + begin[MID], list + begin[HIGH]}, begin[MID], nmid - skip,
          {skip, begin[NCLS] - begin[HIGH]}, g.oplan_have ? kPlanMid : g.ocls_mid};
}

// GraphDev::oplan_list, its order and oplan_fits; ocls_list is there.
static cudaError_t build_out_plan(GraphDev& g, uint64_t padded, int sms, cudaStream_t s) {
  cudaError_t e = g.oplan_list ? cudaSuccess : device_alloc(&g.oplan_list, sizeof(uint32_t) * (g.n ? g.n : 1));
  if (e == cudaSuccess)
    e = build_plan_lists(g.xoff, g.seg_shift, g.n, g.oplan_list, g.oplan_begin, &g.oplan_info, sms, s);
  const bool mixed = padded > 2 * g.oplan_info.low_edges;  // as for the in-edges
  if (e == cudaSuccess && mixed)
    e = sort_by_length(g.xoff, g.seg_shift, g.ocls_list, g.ocls_begin[MID], kLowMax, g.oplan_list, sms, s);
  g.oplan_fits = plan_fits(g.n, g.oplan_begin[MID], g.oplan_info.low_edges, padded);
  g.oplan_built = g.oplan_have = e == cudaSuccess;
  return e;
}

// The persistent loop's rows of a, for graphs up to the lines of persist_fits.
static void take_plan(PullArgs& a, const uint32_t* list, const uint32_t* low, const uint32_t begin[NCLS + 1],
                      bool solo) {
  a.solo = solo;
  a.plan = list;
  a.plan_low = low;
  for (int k = 0; k <= NCLS; ++k) a.plan_begin[k] = begin[k];
}

static cudaError_t launch_pull_persist(PullArgs a, int sms, cudaStream_t s) {
  int per_sm = 0;
  const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pull_persist, 256, 0);
  if (e != cudaSuccess) return e;
  a.list = a.plan;
  for (int k = 0; k <= NCLS; ++k) a.begin[k] = a.plan_begin[k];
  const uint32_t nlow = a.begin[MID] - a.begin[LOW], nmid = a.begin[HIGH] - a.begin[MID],
                 nlong = a.begin[NCLS] - a.begin[HIGH];
  const uint64_t want = std::max<uint64_t>(1, nlong + ((uint64_t)nmid + (nlow + 31) / 32 + 7) / 8);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)std::min<uint64_t>(want, (uint64_t)per_sm * sms));
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeCooperative;
  at.val.cooperative = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_pull_persist, a, a.plan_low);
}

static PullArgs forward_args(const GraphDev& g, const double* t, double alpha) {
  PullArgs a{};
  a.off = g.xtoff;
  a.edg = g.xtedg;
  a.prob = g.pt;
  a.seg = g.xtbase;
  a.shift = g.seg_shift;
  a.list = g.cls_list;
  for (int k = 0; k <= NCLS; ++k) a.begin[k] = g.cls_begin[k];
  a.base = t;
  a.base_scale = 1.0 - alpha;
  a.base_const = 1.0 / (double)g.n;
  a.alpha = alpha;
  a.n = g.n;
  return a;
}

// Jacobi iterations of a from x[0] until the L-inf change is below tol or
// max_iter sweeps; returns the parity holding the answer.
static int pull_loop(prx_context* c, PullArgs& a, const prx_options& o, int* parity, prx_result* res) {
  cudaStream_t s = c->stream;
  a.st = c->st;
  a.xin = nullptr;
  launch_state_reset(c->st, o.max_iterations, o.tolerance, s);
  c->launches += 1;
  if (o.max_iterations > 0 && a.plan && o.loop == PRX_LOOP_AUTO) {
    TRY_CUDA_ST(launch_pull_persist(a, c->sms, s));
    c->launches += 1;
    TRY_CUDA_ST(cudaMemcpyAsync(&c->st_host[1], c->st, sizeof(State), cudaMemcpyDeviceToHost, s));
    TRY_CUDA_ST(cudaStreamSynchronize(s));
    if (c->st_host[1].err & kErrGridWait) FAIL(PRX_ETIMEOUT, "weighted solve: a bounded grid wait ran out");
  } else if (o.max_iterations > 0) {
    for (int k = 1;; k = std::min(2 * k, 16)) {
      for (int i = 0; i < k; ++i) {
        pull_sweep(a, c->sms, s, c->launches);
        k_pull_fin<<<1, 1, 0, s>>>(c->st);
        c->launches += 1;
      }
      TRY_CUDA_ST(cudaGetLastError());
      TRY_CUDA_ST(cudaMemcpyAsync(&c->st_host[1], c->st, sizeof(State), cudaMemcpyDeviceToHost, s));
      TRY_CUDA_ST(cudaStreamSynchronize(s));
      if (c->st_host[1].done) break;
    }
  } else {
    TRY_CUDA_ST(cudaMemcpyAsync(&c->st_host[1], c->st, sizeof(State), cudaMemcpyDeviceToHost, s));
    TRY_CUDA_ST(cudaStreamSynchronize(s));
  }
  *parity = c->st_host[1].iter & 1;
  if (res) {
    res->iterations += c->st_host[1].iter;
    res->last_delta = c->st_host[1].last_delta;
  }
  return PRX_OK;
}

static int weighted_check(prx_context* c, prx_graph* gr, const char* who) {
  if (!c || !gr || gr->ctx != c) {
    set_error(std::string(who) + ": bad context or graph");
    return PRX_EINVAL;
  }
  if (!gr->g.weights_set) {
    set_error(std::string(who) + ": graph has no edge weights (prx_graph_set_weights)");
    return PRX_ESTATE;
  }
  return PRX_OK;
}

static int set_weights(prx_context* c, GraphDev& g, const float* w) {
  cudaStream_t s = c->stream;
  // the arrays stay for the next weights of the same graph version (a batch drops them)
  if (!g.px) TRY_CUDA_ST(device_alloc(&g.px, sizeof(double) * csr_slots(g, g.xseg0, g.xpos)));
  if (!g.pt) TRY_CUDA_ST(device_alloc(&g.pt, sizeof(double) * csr_slots(g, g.xtseg0, g.xtpos)));
  if (!g.wsum) TRY_CUDA_ST(device_alloc(&g.wsum, sizeof(double) * (g.n ? g.n : 1)));
  if (!g.tpos) {
    const cudaError_t e = device_alloc(&g.tpos, sizeof(uint32_t) * csr_slots(g, g.xseg0, g.xpos));
    if (e != cudaErrorMemoryAllocation) TRY_CUDA_ST(e);
  }
  if (!g.wseg && g.nseg > 1) {  // each out-CSR segment's compact start
    TRY_CUDA_ST(device_alloc(&g.wseg, sizeof(unsigned long long) * g.nseg));
    TRY_CUDA_ST(cudaMemcpyAsync(g.wseg, g.xseg0.data(), sizeof(unsigned long long) * g.nseg, cudaMemcpyHostToDevice,
                                s));
  }
  if (!g.oplan_built) {
    if (!g.ocls_list) TRY_CUDA_ST(device_alloc(&g.ocls_list, sizeof(uint32_t) * (g.n ? g.n : 1)));
    uint64_t padded = 0;
    TRY_CUDA_ST(build_class_lists(g.xoff, g.seg_shift, g.n, g.mid_max, g.ocls_list, g.ocls_begin, g.ocls_edges,
                                  c->sms, s, &padded));
    g.ocls_mid = g.mid_max;
    g.oside = g.ocls_edges[LOW] >= 4ull * g.ocls_begin[MID] &&
              (padded <= 2 * g.ocls_edges[LOW] || g.n <= kSideMixed);
    const cudaError_t e = build_out_plan(g, padded, c->sms, s);
    if (e != cudaErrorMemoryAllocation) TRY_CUDA_ST(e);
  }
  launch_state_reset(c->st, 0, 0.0, s);
  if (g.n) {
    const bool found = g.tpos_built;
    const OutRows out = out_rows(g);
    const WeightRows by_class = {out.low, out.mid, out.nlow, out.nmid};
    const uint64_t units = by_class.nmid + (by_class.nlow + (g.oside ? 3ull : 31ull)) / (g.oside ? 4 : 32);
    const int grid = pull_grid(units * 32, 256, c->sms * 8);
    if (g.oside) k_set_weights<8><<<grid, 256, 0, s>>>(weight_csr(g), by_class, w, found, g.wsum, g.px, g.pt, &c->st->err);
    else k_set_weights<1><<<grid, 256, 0, s>>>(weight_csr(g), by_class, w, found, g.wsum, g.px, g.pt, &c->st->err);
    for (int k = 0; k < 2; ++k) {
      const uint32_t nl = out.nlong[k];
      if (!nl) continue;
      k_weight_sums<<<nl, 256, 0, s>>>(weight_csr(g), w, out.longs[k], g.wsum, &c->st->err);
      k_weight_edges<<<dim3(nl, kLongPieces), 256, 0, s>>>(weight_csr(g), w, out.longs[k], found, g.wsum, g.px, g.pt,
                                                          &c->st->err);
    }
  }
  TRY_CUDA_ST(cudaGetLastError());
  TRY_CUDA_ST(cudaMemcpyAsync(&c->st_host[1], c->st, sizeof(State), cudaMemcpyDeviceToHost, s));
  TRY_CUDA_ST(cudaStreamSynchronize(s));
  const uint32_t err = c->st_host[1].err;
  if (err & 1u) FAIL(PRX_EINVAL, "prx_graph_set_weights: every weight must be positive and finite");
  if (err) FAIL(PRX_EINVAL, "prx_graph_set_weights: an out-edge is missing from the in-CSR");
  g.tpos_built = g.tpos != nullptr;
  return PRX_OK;
}

static void opts_or_default(const prx_options* o, prx_options* out) {
  if (o) *out = *o;
  else prx_options_default(out);
}

extern "C" {

int prx_graph_set_weights(prx_context* c, prx_graph* gr, const float* w) {
  if (!c || !gr || gr->ctx != c) FAIL(PRX_EINVAL, "prx_graph_set_weights: bad context or graph");
  GraphDev& g = gr->g;
  if (!g.xoff) FAIL(PRX_ESTATE, "prx_graph_set_weights: graph has no out-CSR");
  if (!w && g.m) FAIL(PRX_EINVAL, "prx_graph_set_weights: weights are NULL");
  TRY_CUDA_ST(cudaSetDevice(c->device));
  g.weights_set = false;
  const int st = set_weights(c, g, w);
  if (st) drop_weights(g);  // whatever failed: no weights, and nothing half allocated for the next call to use
  else g.weights_set = true;
  return st;
}

int prx_solve_weighted(prx_context* c, prx_graph* gr, const double* t, const double* r0, const prx_options* opt,
                       double* r, prx_result* res) {
  int st = weighted_check(c, gr, "prx_solve_weighted");
  if (st) return st;
  prx_options o;
  opts_or_default(opt, &o);
  if (!(o.damping >= 0 && o.damping < 1)) FAIL(PRX_EINVAL, "prx_solve_weighted: damping must be in [0, 1)");
  const GraphDev& g = gr->g;
  prx_result rr{};
  if (g.n == 0) {
    if (res) *res = rr;
    return PRX_OK;
  }
  if (!r) FAIL(PRX_EINVAL, "prx_solve_weighted: r is NULL");
  TRY_CUDA_ST(cudaSetDevice(c->device));
  if ((st = wk_grow(c, 2 * (size_t)g.n))) return st;
  cudaStream_t s = c->stream;
  PullArgs a = forward_args(g, t, o.damping);
  bool plan = persist_fits(g);
  if (plan) TRY_CUDA_ST(ensure_plan(gr->g, c->sms, s, &plan));
  if (plan) take_plan(a, g.plan_list, mixed_lengths(g) ? g.len_list : g.plan_list, g.plan_begin, g.plan_info.solo);
  a.x[0] = c->wk;
  a.x[1] = c->wk + g.n;
  const uint64_t l0 = c->launches;
  TRY_CUDA_ST(cudaEventRecord(c->ev[0], s));
  if (r0) {
    TRY_CUDA_ST(cudaMemcpyAsync(a.x[0], r0, sizeof(double) * g.n, cudaMemcpyDeviceToDevice, s));
  } else if (t) {
    TRY_CUDA_ST(cudaMemcpyAsync(a.x[0], t, sizeof(double) * g.n, cudaMemcpyDeviceToDevice, s));
  } else {
    k_fill<<<pull_grid(g.n, 256, c->sms * 16), 256, 0, s>>>(a.x[0], 1.0 / (double)g.n, g.n);
    c->launches += 1;
  }
  int parity = 0;
  if ((st = pull_loop(c, a, o, &parity, &rr))) return st;
  TRY_CUDA_ST(cudaMemcpyAsync(r, a.x[parity], sizeof(double) * g.n, cudaMemcpyDeviceToDevice, s));
  TRY_CUDA_ST(cudaEventRecord(c->ev[1], s));
  TRY_CUDA_ST(cudaStreamSynchronize(s));
  float ms = 0;
  TRY_CUDA_ST(cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]));
  rr.time_ms = ms;
  rr.computation_time_ms = ms;
  rr.kernel_launches = c->launches - l0;
  if (res) *res = rr;
  return PRX_OK;
}

int prx_adjoint(prx_context* c, prx_graph* gr, const double* t, const double* r, const double* gl,
                const prx_options* opt, double* lambda, double* grad_w, double* grad_t, double* grad_alpha,
                prx_result* res) {
  int st = weighted_check(c, gr, "prx_adjoint");
  if (st) return st;
  prx_options o;
  opts_or_default(opt, &o);
  if (!(o.damping >= 0 && o.damping < 1)) FAIL(PRX_EINVAL, "prx_adjoint: damping must be in [0, 1)");
  const GraphDev& g = gr->g;
  prx_result rr{};
  if (g.n == 0) {
    if (grad_alpha) *grad_alpha = 0.0;
    if (res) *res = rr;
    return PRX_OK;
  }
  if (!r || !gl) FAIL(PRX_EINVAL, "prx_adjoint: r and g are required");
  TRY_CUDA_ST(cudaSetDevice(c->device));
  const int nparts = c->sms * 2;
  if ((st = wk_grow(c, 3 * (size_t)g.n + nparts + 1))) return st;
  cudaStream_t s = c->stream;
  const double alpha = o.damping;
  // lambda = alpha P lambda + g: the pull kernels on the out-CSR
  PullArgs a{};
  a.off = g.xoff;
  a.edg = g.xedg;
  a.prob = g.px;
  a.seg = g.xbase;
  a.shift = g.seg_shift;
  a.list = g.ocls_list;
  for (int k = 0; k <= NCLS; ++k) a.begin[k] = g.ocls_begin[k];
  if (g.oplan_have && g.oplan_fits) take_plan(a, g.oplan_list, g.oplan_list, g.oplan_begin, g.oplan_info.solo);
  a.base = gl;
  a.base_scale = 1.0;
  a.alpha = alpha;
  a.n = g.n;
  a.x[0] = c->wk;
  a.x[1] = c->wk + g.n;
  double* y = c->wk + 2 * (size_t)g.n;
  double* part = c->wk + 3 * (size_t)g.n;
  const uint64_t l0 = c->launches;
  TRY_CUDA_ST(cudaEventRecord(c->ev[0], s));
  TRY_CUDA_ST(cudaMemcpyAsync(a.x[0], gl, sizeof(double) * g.n, cudaMemcpyDeviceToDevice, s));
  int parity = 0;
  if ((st = pull_loop(c, a, o, &parity, &rr))) return st;
  const double* lam = a.x[parity];
  if (lambda) TRY_CUDA_ST(cudaMemcpyAsync(lambda, lam, sizeof(double) * g.n, cudaMemcpyDeviceToDevice, s));
  const int grid = pull_grid((uint64_t)g.n * 32, 256, c->sms * 16);
  if (grad_w) {
    const OutRows out = out_rows(g);
    k_grad_w<<<grid, 256, 0, s>>>(weight_csr(g), g.wsum, r, lam, gl, alpha, g.n, out.mid_max, grad_w);
    c->launches += 1;
    for (int k = 0; k < 2; ++k) {
      const uint32_t nl = out.nlong[k];
      if (!nl) continue;
      k_grad_w_long<<<dim3(nl, kLongPieces), 256, 0, s>>>(weight_csr(g), out.longs[k], g.wsum, r, lam, gl, alpha,
                                                         grad_w);
      c->launches += 1;
    }
  }
  if (grad_t) {
    k_scale<<<pull_grid(g.n, 256, c->sms * 16), 256, 0, s>>>(lam, 1.0 - alpha, g.n, grad_t);
    c->launches += 1;
  }
  if (grad_alpha) {
    PullArgs f = forward_args(g, nullptr, 1.0);  // y = P^T r
    f.base_scale = 0.0;
    f.xin = r;
    f.y = y;
    f.st = nullptr;
    pull_sweep(f, c->sms, s, c->launches);
    k_dot_part<<<nparts, 256, 0, s>>>(lam, y, t, 1.0 / (double)g.n, g.n, part);
    k_dot_final<<<1, 1, 0, s>>>(part, nparts, part + nparts);
    c->launches += 2;
    TRY_CUDA_ST(cudaMemcpyAsync(grad_alpha, part + nparts, sizeof(double), cudaMemcpyDeviceToHost, s));
  }
  TRY_CUDA_ST(cudaEventRecord(c->ev[1], s));
  TRY_CUDA_ST(cudaStreamSynchronize(s));
  TRY_CUDA_ST(cudaGetLastError());
  float ms = 0;
  TRY_CUDA_ST(cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]));
  rr.time_ms = ms;
  rr.computation_time_ms = ms;
  rr.kernel_launches = c->launches - l0;
  if (res) *res = rr;
  return PRX_OK;
}

}  // extern "C"
