// prx_persist.cu -- the whole iteration loop of a small or medium FP64 solve
// as one cooperative kernel.
//
// A sweep of a graph whose arrays fit L2 takes a few microseconds of work,
// but as a CUDA graph body it is four to nine dependent launches (LOW, MID,
// HIGH, hot copy, expansion, finalize, loop condition) with a gap of 3 to 5
// microseconds each.  Here resident blocks iterate by themselves: all three
// in-degree classes in one phase, a grid barrier, the L-inf test by every
// block, and for DF / DF-P the expansion and a second barrier.  The row sums
// are those of prx_update.cu (prx_update.cuh, prx_device.cuh) in the same
// order, so ranks and iteration counts are the same bits.
//
// What bounds it: latency (offsets -> ids -> contributions -> the row's adds
// -> barrier), then the FP64 pipe.
//
// Work split: rows of more than kPlanMid in-edges by
// block (row i to block i mod blocks), the others by warp as units of one
// MID row or 32 LOW rows, counted from the last warp backwards so that the
// blocks that hold long rows get the units of the last round.  LOW rows of
// graphs whose 32-id words mix lengths come in order of length; the words'
// bookkeeping of the dynamic modes is then a pass of its own.  A
// warp keeps what it knows of its first unit (row
// bounds, out-degrees, reciprocals) in registers over the iterations.  Static and ND need no bitmaps; the dynamic
// modes look their rows up with a bit test each instead of queueing them.
//
// Memory: contributions and ranks are written by one block and read by
// others after a grid barrier, so they are read by ordinary loads (never the
// read-only path); the barrier's fences make them visible.  Every wait is
// bounded: a block that runs out sets kErrGridWait and all blocks return.
#include <algorithm>
#include "prx_ctx.h"
#include "prx_update.cuh"

namespace prx {

struct PersistRows {
  const uint32_t* low;   // LOW ids in order of length (GraphDev::len_list)
  const uint32_t* list;  // nmid MID ids, then nlong longer ones (GraphDev::plan_list)
  uint32_t nlow, nmid, nlong;
  bool sorted;           // whether the LOW rows go by `low`, or word by word
  bool solo;             // see WarpShare
};

// Expansion of the changed vertices (nf[p]) into nxt, whichever way
// k_expand_push / k_expand_pull would go.  The out-edges of the changed
// vertices of a word are spread over the warp's lanes, those of out-degree
// above kWarpExpand were queued in xb and get a block each.
constexpr uint32_t kWarpExpand = 1024;

__device__ __forceinline__ void persist_push(const SolveArgs& a, const uint32_t* nf, uint32_t* nxt, uint32_t nbig,
                                             uint32_t warp, uint32_t warps) {
  const uint32_t words = (a.n + 31) >> 5, lane = lane_id();
  for (uint32_t w = warp; w < words; w += warps) {
    const uint32_t word = nf[w];
    if (!word) continue;
    uint32_t b = 0, len = 0;
    if ((word >> lane) & 1u) {
      const uint32_t u = (w << 5) | lane;
      b = a.xoff[u];
      len = a.xoff[u + 1] - b;
      // queued, by the degree given with the graph, which may differ from the row's
      if (len > kWarpExpand && __ldg(a.xtdat + u) > kWarpExpand) len = 0;
    }
    uint32_t incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if ((int)lane >= o) incl += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    const uint32_t base = b - (incl - len);  // edge of flat index t: base of its owner + t
    for (uint32_t t0 = 0; t0 < total; t0 += 32) {
      const uint32_t t = t0 + lane;
      uint32_t own = 0;  // the first lane whose inclusive sum exceeds t
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        const uint32_t y = __shfl_sync(0xffffffffu, incl, own + o - 1);
        if (y <= t) own += o;
      }
      own = min(own, 31u);
      const uint32_t at = __shfl_sync(0xffffffffu, base, own);
      if (t < total) set_bit(nxt, __ldg(a.xedg + (uint32_t)(at + t)));
    }
  }
  for (uint32_t i = blockIdx.x; i < nbig; i += gridDim.x) {
    const uint32_t u = a.xb[i], e = a.xoff[u + 1];
    for (uint32_t j = a.xoff[u] + threadIdx.x; j < e; j += blockDim.x) set_bit(nxt, __ldg(a.xedg + j));
  }
}

// LOW rows by lane; MID and HIGH rows by warp, 128 ids a step, so that a long
// row without a changed source does not hold one lane up.
__device__ __forceinline__ void persist_pull(const SolveArgs& a, const PersistRows& rows, const uint32_t* nf,
                                             uint32_t* nxt, uint32_t warp, uint32_t warps) {
  const uint32_t words = (a.n + 31) >> 5, lane = lane_id();
  for (uint32_t i = warp; i < rows.nmid + rows.nlong; i += warps) {
    const uint32_t v = rows.list[i];
    if ((nxt[v >> 5] >> (v & 31u)) & 1u) continue;
    const uint32_t e = a.xtoff[v + 1];
    bool hit = false;
    for (uint32_t j = a.xtoff[v]; j < e && !hit; j += 128) {
      uint32_t bits = 0;
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t u = __ldg(a.xtedg + min(j + lane + 32 * k, e - 1));
        bits |= nf[u >> 5] >> (u & 31u);
      }
      hit = __any_sync(0xffffffffu, bits & 1u);
    }
    if (hit && lane == 0) set_bit(nxt, v);
  }
  for (uint32_t w = warp; w < words; w += warps) {
    const uint32_t todo = a.low_bm[w] & ~nxt[w];
    const uint32_t v = (w << 5) | lane;
    bool hit = false;
    if (v < a.n && ((todo >> lane) & 1u)) {
      const uint32_t e = a.xtoff[v + 1];
      for (uint32_t j = a.xtoff[v]; j < e && !hit; j += 4) {
        uint32_t bits = 0;
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
          const uint32_t u = __ldg(a.xtedg + min(j + k, e - 1));
          bits |= nf[u >> 5] >> (u & 31u);
        }
        hit = bits & 1u;
      }
    }
    const unsigned add = __ballot_sync(0xffffffffu, hit);
    if (lane == 0 && add) atomicOr(&nxt[w], add);
  }
}

// A unit's rows as a warp knows them: the MID row in every lane, or lane i's
// LOW row.
struct Unit {
  uint32_t v, s, e;   // row v, its in-edges [s, e)
  bool row;           // this lane has one
  uint32_t d;         // out-degree
  uint64_t R;         // its reciprocal (load_vertex)
};

// Three blocks per SM (80 registers): what a unit waits for counts more here
// than how many are in flight.  K: see warp_row_sums.
template <int MODE, int K>
__global__ void __launch_bounds__(kThreads, 3) k_persist(SolveArgs a, PersistRows rows) {
  using T = ModeTraits<MODE>;
  __shared__ double part[256];
  __shared__ double s_tree[kThreads / 32][RowTree::kSlots];
  __shared__ unsigned long long s_el;
  __shared__ uint32_t s_nf, s_xb, s_marked;
  State* st = a.st;
  if (st->done) return;
  const uint32_t lane = lane_id(), t = threadIdx.x;
  const RowTree tree{s_tree[t >> 5]};
  const WarpShare share(rows.nlong, rows.solo);
  const uint32_t warps = share.warps, warp = share.warp;
  const uint32_t words = (a.n + 31) >> 5;
  const uint32_t units = rows.nmid + (rows.sorted ? (rows.nlow + 31) / 32 : words);
  const int max_iter = st->max_iter;
  const double tol = st->tol;
  unsigned long long edges = 0;
  auto load_unit = [&](uint32_t u) {
    Unit x{};
    if (u < rows.nmid) {
      x.v = __ldg(rows.list + u);
      x.row = true;
    } else if (rows.sorted) {
      const uint32_t i = 32 * (u - rows.nmid) + lane;
      x.row = i < rows.nlow;
      x.v = x.row ? __ldg(rows.low + i) : 0u;
    } else {
      const uint32_t w = u - rows.nmid;
      x.v = (w << 5) | lane;
      x.row = x.v < a.n && ((__ldg(a.low_bm + w) >> lane) & 1u);
    }
    if (x.row) {
      x.s = __ldg(a.xtoff + x.v);
      x.e = __ldg(a.xtoff + x.v + 1);
      x.d = __ldg(a.xtdat + x.v);
      x.R = x.d < kQuotTable ? __ldg(a.qtab + x.d) : 0ull;
    }
    return x;
  };
  // this warp's first unit of LOW rows
  const uint32_t low0 = warp < rows.nmid ? warp + (rows.nmid - warp + warps - 1) / warps * warps : warp;
  // the unit this warp takes next: loaded while the one before it is summed,
  // over the end of an iteration too (what a unit holds does not change)
  Unit coming{};
  if (warp < units) coming = load_unit(warp);
  auto take = [&](uint32_t u) {
    const Unit x = coming;
    if (units > warps) coming = load_unit(u + warps < units ? u + warps : warp);
    return x;
  };
  GridBarrier bar(st);
  for (int it = 0;; ++it) {
    const int p = it & 1;
    const double* c = a.c[p];
    const uint32_t* cur = T::DYN ? a.bm[it % 3] : nullptr;
    uint32_t* nxt = T::DYN ? a.bm[(it + 1) % 3] : nullptr;
    uint32_t* prev = T::DYN ? a.bm[(it + 2) % 3] : nullptr;
    unsigned long long emax = 0;
    unsigned int mag = 0;
    uint32_t marked = 0;
    auto affected = [&](uint32_t v) { return !T::DYN || ((cur[v >> 5] >> (v & 31u)) & 1u); };
    // one vertex, by the thread that holds its sum
    auto finish_one = [&](uint32_t v, double x, uint32_t len, const VertexIn& in) {
      bool survive, changed;
      const unsigned long long ev = finish_vertex<MODE>(a, v, x, p, survive, changed, mag, in);
      emax = ev > emax ? ev : emax;
      edges += len;
      if (T::DYN && survive) atomicOr(&nxt[v >> 5], 1u << (v & 31u));
      if (T::FRONTIER && changed && (T::PRUNE || test_and_set(a.naff, v))) {  // see fresh_changes
        atomicOr(&a.nf[p][v >> 5], 1u << (v & 31u));
        count_one(&st->pnf[it % 3]);
        if (in.d > kWarpExpand) a.xb[atomicAdd(&st->pxb[it % 3], 1u)] = v;
      }
    };
    // a word's bookkeeping in the dynamic modes; returns its affected vertices
    auto word_pass = [&](uint32_t w) -> uint32_t {
      const uint32_t v = (w << 5) | lane;
      const uint32_t cw = cur[w], pw = prev[w];
      __syncwarp();  // every lane has read prev[w] before lane 0 clears it
      if (T::FRONTIER && lane == 0) marked += __popc(cw);
      if (((pw & ~cw) >> lane) & 1u) {  // updated last iteration, not this one: refresh parity p^1
        a.r[p ^ 1][v] = a.r[p][v];
        a.c[p ^ 1][v] = c[v];
      }
      if (lane == 0) {
        if (pw) prev[w] = 0;  // becomes the empty nxt of the next iteration
        if (T::FRONTIER && a.nf[p ^ 1][w]) a.nf[p ^ 1][w] = 0;
      }
      return cw;
    };
    for (uint32_t i = share.row; i < rows.nlong; i += gridDim.x) {
      const uint32_t v = __ldg(rows.list + rows.nmid + i);
      if (!affected(v)) continue;
      const uint32_t s = __ldg(a.xtoff + v), d = __ldg(a.xtoff + v + 1) - s;
      const VertexIn in = load_vertex(a, v, p);
      const double x = high_row_sum<double, true, true>(c, a.xtedg + s, d, t, part);
      if (t == 0) finish_one(v, x, d, in);
    }
    // four MID rows are folded and finished together (see RowTree); lane k
    // keeps what row k needs
    uint32_t qv = 0, qlen = 0, held = 0;
    VertexIn qin{};
    auto flush = [&] {
      double z = tree.fold<true>(held);
      z = __shfl_sync(0xffffffffu, z, (lane & 3u) * 8);
      if (lane < held) finish_one(qv, z, qlen, qin);
      held = 0;
    };
    for (uint32_t u = warp; u < rows.nmid; u += warps) {
      const Unit x = take(u);
      if (!affected(x.v)) continue;
      if (lane == held) {
        qv = x.v;
        qlen = x.e - x.s;
        qin = {x.d, x.R, a.r[p][x.v]};
      }
      bool bad = false;
      const double sum = mid_lane_sums<double, true, true, true>(c, a.xtedg + x.s, x.e - x.s, lane, bad);
      if (__any_sync(0xffffffffu, bad)) {  // terms out of soft_add's range: this row by FP64 adds alone
        const double y = mid_row_sum_plain<true>(c, a.xtedg + x.s, x.e - x.s, lane);
        if (lane == 0) finish_one(x.v, y, x.e - x.s, VertexIn{x.d, x.R, a.r[p][x.v]});
        continue;
      }
      tree.put(held++, sum);
      if (held == RowTree::kRows) flush();
    }
    if (held) flush();
    for (uint32_t u = low0; u < units; u += warps) {
      const Unit x = take(u);
      bool mine = x.row;
      if (T::DYN) {
        if (rows.sorted) {
          mine = mine && affected(x.v);
        } else {
          const uint32_t cw = word_pass(u - rows.nmid);  // every lane: MID rows have stale copies too
          mine = mine && ((cw >> lane) & 1u);
        }
        if (!__any_sync(0xffffffffu, mine)) continue;
      }
      VertexIn in = {x.d, x.R, 0.0};
      if (mine) in.r = a.r[p][x.v];
      const double sum = warp_row_sums<true, true, 1, K>(c, a.xtedg, x.s, mine ? x.e : x.s, 0.0, nullptr, false);
      if (!T::DYN || rows.sorted) {
        if (mine) finish_one(x.v, sum, x.e - x.s, in);
        continue;
      }
      // the lanes are one word: its bits go out together
      bool survive = false, changed = false;
      if (mine) {
        const unsigned long long ev = finish_vertex<MODE>(a, x.v, sum, p, survive, changed, mag, in);
        emax = ev > emax ? ev : emax;
        edges += x.e - x.s;
      }
      const uint32_t w = u - rows.nmid;
      const unsigned keep = __ballot_sync(0xffffffffu, mine && survive);
      if (lane == 0 && keep) atomicOr(&nxt[w], keep);
      if (T::FRONTIER) {
        const unsigned chg = fresh_changes<T::PRUNE>(a.naff, w, __ballot_sync(0xffffffffu, mine && changed), lane);
        if (chg) {
          if (lane == 0) {
            atomicOr(&a.nf[p][w], chg);
            atomicAdd(&st->pnf[it % 3], (uint32_t)__popc(chg));
          }
          if (((chg >> lane) & 1u) && in.d > kWarpExpand) push(a.xb, &st->pxb[it % 3], x.v);
        }
      }
    }
    if (T::DYN && rows.sorted)
      for (uint32_t w = warp; w < words; w += warps) word_pass(w);
    block_max_bits(emax, &st->pel[it % 3]);
    if (T::FRONTIER) block_sum_u32(marked, &st->pmarked[it % 3]);
    if (blockIdx.x == 0 && t == 0) {  // the next iteration's slots (last read two barriers ago)
      st->pel[(it + 1) % 3] = 0;
      if (T::FRONTIER) st->pnf[(it + 1) % 3] = st->pxb[(it + 1) % 3] = st->pmarked[(it + 1) % 3] = 0;
    }
    if (!bar.sync([&] {
          s_el = *(volatile unsigned long long*)&st->pel[it % 3];
          if (T::FRONTIER) {
            s_nf = *(volatile uint32_t*)&st->pnf[it % 3];
            s_xb = *(volatile uint32_t*)&st->pxb[it % 3];
            s_marked = *(volatile uint32_t*)&st->pmarked[it % 3];
          }
        }))
      return;
    const double el = __longlong_as_double((long long)s_el);
    if (el < tol || it + 1 >= max_iter) {  // pagerankLoopCuU :680,689
      if (blockIdx.x == 0 && t == 0) {
        st->iter = it + 1;
        st->last_delta = el;
        st->done = 1;
      }
      break;
    }
    if (T::FRONTIER && s_nf) {  // no vertex to expand: no second barrier either
      if (expand_by_pull(s_nf, s_marked, a.n, a.pull_threshold)) persist_pull(a, rows, a.nf[p], nxt, share.any, share.all);
      else persist_push(a, a.nf[p], nxt, s_xb, share.any, share.all);
      if (!bar.sync([] {})) return;
    }
  }
  if (T::DYN) block_sum_u64(edges, &st->edges);
}

// ---- FP32 refinement ------------------------------------------------------------
// Sum of ce[edg[j]], j in [s, e), front to back: eight gathers in flight; ids
// outside the row in its first and last groups give +0, which changes no sum
// that started at +0.
__device__ __forceinline__ float lane_row_sum32(const float* ce, const uint32_t* __restrict__ edg, uint32_t s,
                                                uint32_t e) {
  float acc = 0.f;
  if (s >= e) return acc;
  auto ids = [&](uint32_t j) {
    return j < e ? __ldg(reinterpret_cast<const uint4*>(edg + j)) : make_uint4(0, 0, 0, 0);
  };
  uint32_t j = s & ~3u;
  uint4 g0 = ids(j), g1 = ids(j + 4);
  for (; j < e; j += 8) {
    const uint32_t u[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
    float x[8];
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) x[k] = j + k >= s && j + k < e ? ce[u[k]] : 0.f;
    g0 = ids(j + 8);
    g1 = ids(j + 12);
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) acc += x[k];
  }
  return acc;
}

// The whole loop of prx_refine.cu (round 0 on the initial ranks, then FP64
// residual sweeps and FP32 rounds) on the same units; the sums and the tests
// that end a round are those of the launched kernels, the same bits.  Rows of
// 1025 to mid_max ids, which a warp of the launched sweep sums alone, have their
// terms brought in by a block.  Whole solves, launched | here, ms: R-MAT 2^10 1.62
// | 0.40, 2^16 2.66 | 0.67, 2^18 3.67 | 1.46, 2^20 9.0 | 5.7, 2^22 27.9 | 25.1,
// web-like 30k 0.39 | 0.12, 200k 0.56 | 0.36, 1.5M 2.00 | 1.71, grid 500^2 0.50 |
// 0.21, 1000^2 0.57 | 0.35.  What bounds it: as k_persist, then L1 and L2 sectors
// of the gathers.
constexpr uint32_t kRowVals = 2048;

template <int K>
__global__ void __launch_bounds__(kThreads, 3) k_persist_refine(SolveArgs a, PersistRows rows) {
  __shared__ double part[256];
  __shared__ float vals[kRowVals];
  __shared__ double s_tree[kThreads / 32][RowTree::kSlots];
  __shared__ unsigned long long s_el;
  __shared__ uint32_t s_dl, s_em;
  State* st = a.st;
  if (st->done) return;
  const uint32_t lane = lane_id(), t = threadIdx.x;
  const RowTree tree{s_tree[t >> 5]};
  const WarpShare share(rows.nlong, rows.solo);
  const uint32_t warps = share.warps, warp = share.warp;
  const uint32_t words = (a.n + 31) >> 5;
  const uint32_t units = rows.nmid + (rows.sorted ? (rows.nlow + 31) / 32 : words);
  const int max_iter = st->max_iter;
  const double tol = st->tol;
  const float P32 = (float)a.P, tol32 = (float)tol;
  auto load_unit = [&](uint32_t u) {
    Unit x{};
    if (u < rows.nmid) {
      x.v = __ldg(rows.list + u);
      x.row = true;
    } else if (rows.sorted) {
      const uint32_t i = 32 * (u - rows.nmid) + lane;
      x.row = i < rows.nlow;
      x.v = x.row ? __ldg(rows.low + i) : 0u;
    } else {
      const uint32_t w = u - rows.nmid;
      x.v = (w << 5) | lane;
      x.row = x.v < a.n && ((__ldg(a.low_bm + w) >> lane) & 1u);
    }
    if (x.row) {
      x.s = __ldg(a.xtoff + x.v);
      x.e = __ldg(a.xtoff + x.v + 1);
      x.d = __ldg(a.xtdat + x.v);
    }
    return x;
  };
  const uint32_t low0 = warp < rows.nmid ? warp + (rows.nmid - warp + warps - 1) / warps * warps : warp;
  Unit coming{};  // as in k_persist
  if (warp < units) coming = load_unit(warp);
  auto take = [&](uint32_t u) {
    const Unit x = coming;
    if (units > warps) coming = load_unit(u + warps < units ? u + warps : warp);
    return x;
  };
  GridBarrier bar(st);
  int slot = 0;  // of the sweep's maxima
  auto next_slot = [&] {  // cleared a sweep ahead (last read two barriers ago)
    if (blockIdx.x == 0 && t == 0) {
      const int z = (slot + 1) % 3;
      st->pel[z] = 0;
      st->pnf[z] = st->pmarked[z] = 0;
    }
  };

  // FP64 residual sweep of the base ranks
  auto sweep64 = [&]() -> bool {
    const double* c = a.c[0];
    unsigned long long emax = 0;
    unsigned int mag = 0;
    auto finish_one = [&](uint32_t v, double x, const VertexIn& in) {
      bool survive, changed;
      const unsigned long long ev = finish_vertex<MODE_REFINE64>(a, v, x, 0, survive, changed, mag, in);
      emax = ev > emax ? ev : emax;
    };
    for (uint32_t i = share.row; i < rows.nlong; i += gridDim.x) {
      const uint32_t v = __ldg(rows.list + rows.nmid + i);
      const uint32_t s = __ldg(a.xtoff + v), d = __ldg(a.xtoff + v + 1) - s;
      const VertexIn in{__ldg(a.xtdat + v), 0ull, a.r[0][v]};
      const double x = high_row_sum<double, true, true>(c, a.xtedg + s, d, t, part);
      if (t == 0) finish_one(v, x, in);
    }
    uint32_t qv = 0, held = 0;
    VertexIn qin{};
    auto flush = [&] {
      double z = tree.fold<true>(held);
      z = __shfl_sync(0xffffffffu, z, (lane & 3u) * 8);
      if (lane < held) finish_one(qv, z, qin);
      held = 0;
    };
    for (uint32_t u = warp; u < rows.nmid; u += warps) {
      const Unit x = take(u);
      const VertexIn in{x.d, 0ull, a.r[0][x.v]};
      if (lane == held) {
        qv = x.v;
        qin = in;
      }
      bool bad = false;
      const double sum = mid_lane_sums<double, true, true, true>(c, a.xtedg + x.s, x.e - x.s, lane, bad);
      if (__any_sync(0xffffffffu, bad)) {
        const double y = mid_row_sum_plain<true>(c, a.xtedg + x.s, x.e - x.s, lane);
        if (lane == 0) finish_one(x.v, y, in);
        continue;
      }
      tree.put(held++, sum);
      if (held == RowTree::kRows) flush();
    }
    if (held) flush();
    for (uint32_t u = low0; u < units; u += warps) {
      const Unit x = take(u);
      VertexIn in{x.d, 0ull, 0.0};
      if (x.row) in.r = a.r[0][x.v];
      const double sum = warp_row_sums<true, true, 1, K>(c, a.xtedg, x.s, x.e, 0.0, nullptr, false);
      if (x.row) finish_one(x.v, sum, in);
    }
    block_max_bits(emax, &st->pel[slot]);
    next_slot();
    const bool ok = bar.sync([&] { s_el = *(volatile unsigned long long*)&st->pel[slot]; });
    slot = (slot + 1) % 3;
    return ok;
  };

  // FP32 sweep of the correction, parity q
  auto sweep32 = [&](int q) -> bool {
    const float* ce = a.ce[q];
    unsigned int emax = 0, mag = 0;
    auto finish_one = [&](uint32_t v, float sum, uint32_t d, float rho, float old) {
      const float en = fmaf(P32, sum, rho);
      a.e[q ^ 1][v] = en;
      a.ce[q ^ 1][v] = __fdividef(en, (float)d);
      emax = max(emax, __float_as_uint(fabsf(en - old)));
      mag = max(mag, __float_as_uint(fabsf(en)));
    };
    for (uint32_t i = share.row; i < rows.nlong; i += gridDim.x) {
      const uint32_t v = __ldg(rows.list + rows.nmid + i);
      const uint32_t s = __ldg(a.xtoff + v), d = __ldg(a.xtoff + v + 1) - s;
      const uint32_t* __restrict__ ed = a.xtedg + s;
      float acc = 0.f;
      if (d > a.mid_max) {
#pragma unroll 8
        for (uint32_t j = t; j < d; j += kThreads) acc += ce[__ldg(ed + j)];
      } else {  // 32 sums, their terms brought in by the whole block
        for (uint32_t j0 = 0; j0 < d; j0 += kRowVals) {
#pragma unroll
          for (uint32_t j = t; j < kRowVals; j += kThreads) vals[j] = j0 + j < d ? ce[__ldg(ed + j0 + j)] : 0.f;
          __syncthreads();
          if (t < 32) {
#pragma unroll 16
            for (uint32_t j = lane; j < kRowVals; j += 32) acc += vals[j];
          }
          __syncthreads();
        }
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
      if (d > a.mid_max) {
        if (lane == 0) vals[t >> 5] = acc;
        __syncthreads();
        if (t < 32) {
          acc = t < 8 ? vals[t] : 0.f;
#pragma unroll
          for (int o = 4; o; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        }
        __syncthreads();
      }
      if (t == 0) finish_one(v, acc, __ldg(a.xtdat + v), a.rho[v], a.e[q][v]);
    }
    for (uint32_t u = warp; u < rows.nmid; u += warps) {
      const Unit x = take(u);
      const float rho = a.rho[x.v], old = a.e[q][x.v];
      const uint32_t* __restrict__ ed = a.xtedg + x.s;
      const uint32_t d = x.e - x.s;
      float acc = 0.f;
      for (uint32_t j0 = 0; j0 < d; j0 += 256) {
        float y[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
          const uint32_t j = j0 + 32 * k + lane;
          y[k] = j < d ? ce[__ldg(ed + j)] : 0.f;
        }
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) acc += y[k];
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
      if (lane == 0) finish_one(x.v, acc, x.d, rho, old);
    }
    for (uint32_t u = low0; u < units; u += warps) {
      const Unit x = take(u);
      if (!x.row) continue;
      const float rho = a.rho[x.v], old = a.e[q][x.v];
      finish_one(x.v, lane_row_sum32(ce, a.xtedg, x.s, x.e), x.d, rho, old);
    }
    block_max_u32(emax, &st->pnf[slot]);
    block_max_u32(mag, &st->pmarked[slot]);
    next_slot();
    const bool ok = bar.sync([&] {
      s_dl = *(volatile uint32_t*)&st->pnf[slot];
      s_em = *(volatile uint32_t*)&st->pmarked[slot];
    });
    slot = (slot + 1) % 3;
    return ok;
  };

  const uint32_t v0 = blockIdx.x * blockDim.x + t, stride = gridDim.x * blockDim.x;
  const float c0 = (float)a.C0;
  for (uint32_t v = v0; v < a.n; v += stride) {  // round 0: x_b = 0, rho = C0, e_0 = the initial ranks
    const float x = (float)a.r[0][v];
    a.r[0][v] = 0.0;
    a.rho[v] = c0;
    a.e[0][v] = x;
    a.ce[0][v] = __fdividef(x, (float)__ldg(a.xtdat + v));
  }
  if (!bar.sync([] {})) return;
  int iter = 0, rounds = 0;
  double el = 0.0;
  bool done = false;
  for (;;) {
    float prev = 0.f, prev2 = 0.f;
    int k32 = 0;
    for (bool more = true; more;) {
      if (!sweep32(k32 & 1)) return;
      const float dl = __uint_as_float(s_dl), em = __uint_as_float(s_em);
      ++iter;
      ++k32;
      more = !(dl < tol32 || dl < em * 0x1p-18f || iter >= max_iter || fp32_round_done(dl, prev, prev2, tol));
      prev2 = prev;
      prev = dl;
    }
    const float* e = a.e[k32 & 1];
    for (uint32_t v = v0; v < a.n; v += stride) {  // x_b += e
      const double x = a.r[0][v] + (double)e[v];
      a.r[0][v] = x;
      a.c[0][v] = div_count(x, __ldg(a.xtdat + v), __ldg(a.rcp + v));
    }
    if (iter >= max_iter) break;
    if (!bar.sync([] {}) || !sweep64()) return;
    el = __longlong_as_double((long long)s_el);
    ++iter;
    ++rounds;
    if (el < tol || iter >= max_iter) {
      done = true;
      break;
    }
  }
  if (blockIdx.x == 0 && t == 0) {
    st->iter = iter;
    st->rounds = rounds;
    st->last_delta = el;
    st->done = done;
  }
}

// Cooperative launch of `want` blocks, or as many as are resident.
template <class... A>
static cudaError_t launch_resident(void (*kernel)(A...), uint64_t want, int threads, int sms, cudaStream_t s,
                                   A... args) {
  int per_sm = 0;  // resident blocks per SM of this build
  const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)std::min<uint64_t>(want, (uint64_t)per_sm * sms));
  cfg.blockDim = dim3(threads);
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeCooperative;
  at.val.cooperative = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <int MODE, int K>
static cudaError_t persist_k(const SolveArgs& a, const PersistRows& rows, uint64_t want, int threads, int sms,
                             cudaStream_t s) {
  return launch_resident(k_persist<MODE, K>, want, threads, sms, s, a, rows);
}
template <int MODE>
static cudaError_t persist_t(const SolveArgs& a, const PersistRows& rows, int sms, cudaStream_t s) {
  // a warp per unit and a block per long row; no more blocks than are resident
  const uint64_t units = (uint64_t)rows.nmid + ((uint64_t)(rows.sorted ? rows.nlow : a.n) + 31) / 32;
  // A few units go to more SMs in smaller blocks (long rows need 256
  // threads): the warps of an SM share its FP64 pipe.
  const int threads = rows.nlong || units > 4ull * sms ? kThreads : units > 2ull * sms ? 128 : 64;
  const uint64_t per = threads / 32;
  const uint64_t want = std::max<uint64_t>(1, rows.nlong + (units + per - 1) / per);
  // two of four adds on the integer pipes (one gives 2% less on a web-like
  // graph of 1.5M vertices); four warps an SM leave its FP64 pipe idle for
  // the latency of their adds (R-MAT 2^13: 6.4 us an iteration without, 7.2 with)
  return a.int_adds && units > 4ull * sms ? persist_k<MODE, 2>(a, rows, want, threads, sms, s)
                                          : persist_k<MODE, 0>(a, rows, want, threads, sms, s);
}

static PersistRows persist_rows(const GraphDev& g) {
  return {g.len_list, g.plan_list + g.plan_begin[MID], g.plan_begin[MID], g.plan_begin[HIGH] - g.plan_begin[MID],
          g.plan_begin[NCLS] - g.plan_begin[HIGH], mixed_lengths(g), g.plan_info.solo};
}

cudaError_t launch_persist_refine(const SolveArgs& a, const GraphDev& g, int sms, cudaStream_t s) {
  const PersistRows rows = persist_rows(g);
  const uint64_t units = (uint64_t)rows.nmid + ((uint64_t)(rows.sorted ? rows.nlow : a.n) + 31) / 32;
  const uint64_t want = std::max<uint64_t>(1, rows.nlong + (units + kThreads / 32 - 1) / (kThreads / 32));
  return a.int_adds ? launch_resident(k_persist_refine<2>, want, kThreads, sms, s, a, rows)
                    : launch_resident(k_persist_refine<0>, want, kThreads, sms, s, a, rows);
}

cudaError_t launch_persist(const SolveArgs& a, const GraphDev& g, int mode, int sms, cudaStream_t s) {
  const PersistRows rows = persist_rows(g);
  switch (mode) {
    case PRX_DYNAMIC_TRAVERSAL: return persist_t<PRX_DYNAMIC_TRAVERSAL>(a, rows, sms, s);
    case PRX_DYNAMIC_FRONTIER: return persist_t<PRX_DYNAMIC_FRONTIER>(a, rows, sms, s);
    case PRX_PRUNE_DYNAMIC_FRONTIER: return persist_t<PRX_PRUNE_DYNAMIC_FRONTIER>(a, rows, sms, s);
    default: return persist_t<PRX_STATIC>(a, rows, sms, s);
  }
}

}  // namespace prx
