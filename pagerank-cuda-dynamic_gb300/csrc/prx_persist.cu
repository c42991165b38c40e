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
// Work split: HIGH rows by block (block b takes rows b, b + blocks, ...),
// MID rows and 32-id words of LOW rows by warp, counted from the last warp
// backwards so that the blocks that hold HIGH rows get the units of the last
// round.  Static and ND need no bitmaps; the dynamic modes look their MID and
// HIGH rows up in the static class lists (a bit test each) instead of
// queueing them.
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
  uint32_t mid, nmid;    // MID rows: cls_list[mid .. mid + nmid)
  uint32_t high, nhigh;  // HIGH rows
};

// Expansion of the changed vertices (nf[p]) into nxt, whichever way
// k_expand_push / k_expand_pull would go.  The out-edges of the changed
// vertices of a word are spread over the warp's lanes, those of more than
// kWarpExpand out-edges were queued in xb and get a block each.
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
      if (len > kWarpExpand) len = 0;  // queued
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
  // MID and HIGH lie side by side in cls_list
  for (uint32_t i = warp; i < rows.nmid + rows.nhigh; i += warps) {
    const uint32_t v = a.cls_list[rows.mid + i];
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

template <int MODE>
__global__ void __launch_bounds__(kThreads, 4) k_persist(SolveArgs a, PersistRows rows) {
  using T = ModeTraits<MODE>;
  __shared__ double part[256];
  __shared__ unsigned long long s_el;
  __shared__ uint32_t s_nf, s_xb, s_marked;
  State* st = a.st;
  if (st->done) return;
  const uint32_t lane = lane_id(), t = threadIdx.x;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t warp = warps - 1 - ((blockIdx.x * blockDim.x + t) >> 5);
  const uint32_t words = (a.n + 31) >> 5;
  const uint32_t w0 = (warp + warps - rows.nmid % warps) % warps;
  const int max_iter = st->max_iter;
  const double tol = st->tol;
  unsigned long long edges = 0;
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
    // one MID / HIGH vertex, by the thread that holds its sum
    auto finish_one = [&](uint32_t v, double x, uint32_t d) {
      bool survive, changed;
      const unsigned long long ev = finish_vertex<MODE>(a, v, x, p, survive, changed, mag);
      emax = ev > emax ? ev : emax;
      edges += d;
      if (T::DYN && survive) atomicOr(&nxt[v >> 5], 1u << (v & 31u));
      if (T::FRONTIER && changed && (T::PRUNE || test_and_set(a.naff, v))) {  // see fresh_changes
        atomicOr(&a.nf[p][v >> 5], 1u << (v & 31u));
        atomicAdd(&st->pnf[it % 3], 1u);
        if (a.xtdat[v] > kWarpExpand) a.xb[atomicAdd(&st->pxb[it % 3], 1u)] = v;
      }
    };
    for (uint32_t i = blockIdx.x; i < rows.nhigh; i += gridDim.x) {
      const uint32_t v = a.cls_list[rows.high + i];
      if (T::DYN && !((cur[v >> 5] >> (v & 31u)) & 1u)) continue;
      const uint32_t s = a.xtoff[v], d = a.xtoff[v + 1] - s;
      const double x = high_row_sum<double, true>(c, a.xtedg + s, d, t, part);
      if (t == 0) finish_one(v, x, d);
    }
    for (uint32_t i = warp; i < rows.nmid; i += warps) {
      const uint32_t v = a.cls_list[rows.mid + i];
      if (T::DYN && !((cur[v >> 5] >> (v & 31u)) & 1u)) continue;
      const uint32_t s = a.xtoff[v], d = a.xtoff[v + 1] - s;
      const double x = mid_row_sum<double, true>(c, a.xtedg + s, d, lane);
      if (lane == 0) finish_one(v, x, d);
    }
    for (uint32_t w = w0; w < words; w += warps) {
      const uint32_t v = (w << 5) | lane;
      bool mine = v < a.n && ((a.low_bm[w] >> lane) & 1u);
      if (T::DYN) {
        const uint32_t cw = cur[w], pw = prev[w];
        if (T::FRONTIER && lane == 0) marked += __popc(cw);
        if (((pw & ~cw) >> lane) & 1u) {  // updated last iteration, not this one: refresh parity p^1
          a.r[p ^ 1][v] = a.r[p][v];
          a.c[p ^ 1][v] = c[v];
        }
        if (lane == 0) {
          if (pw) prev[w] = 0;  // becomes the empty nxt of the next iteration
          if (T::FRONTIER && a.nf[p ^ 1][w]) a.nf[p ^ 1][w] = 0;
        }
        mine = mine && ((cw >> lane) & 1u);
        if (!__any_sync(0xffffffffu, mine)) continue;
      }
      const uint32_t s = mine ? a.xtoff[v] : 0, e = mine ? a.xtoff[v + 1] : 0;
      const double sum = warp_row_sums<true>(c, a.xtedg, s, e, 0.0, nullptr, false, a.int_adds);
      bool survive = false, changed = false;
      if (mine) {
        const unsigned long long ev = finish_vertex<MODE>(a, v, sum, p, survive, changed, mag);
        emax = ev > emax ? ev : emax;
        edges += e - s;
      }
      if (T::DYN) {
        const unsigned keep = __ballot_sync(0xffffffffu, mine && survive);
        if (lane == 0 && keep) atomicOr(&nxt[w], keep);
      }
      if (T::FRONTIER) {
        const unsigned chg = fresh_changes<T::PRUNE>(a.naff, w, __ballot_sync(0xffffffffu, mine && changed), lane);
        if (chg) {
          if (lane == 0) {
            atomicOr(&a.nf[p][w], chg);
            atomicAdd(&st->pnf[it % 3], (uint32_t)__popc(chg));
          }
          if (((chg >> lane) & 1u) && a.xtdat[v] > kWarpExpand) push(a.xb, &st->pxb[it % 3], v);
        }
      }
    }
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
      if (expand_by_pull(s_nf, s_marked, a.n, a.pull_threshold)) persist_pull(a, rows, a.nf[p], nxt, warp, warps);
      else persist_push(a, a.nf[p], nxt, s_xb, warp, warps);
      if (!bar.sync([] {})) return;
    }
  }
  if (T::DYN) block_sum_u64(edges, &st->edges);
}

template <int MODE>
static cudaError_t persist_t(const SolveArgs& a, const PersistRows& rows, int sms, int* per_sm, cudaStream_t s) {
  if (!*per_sm) {
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_persist<MODE>, kThreads, 0);
    if (e != cudaSuccess) return e;
  }
  // a warp per MID row and 32-id word, a block per HIGH row; no more blocks than are resident
  const uint64_t units = (uint64_t)rows.nmid + ((uint64_t)a.n + 31) / 32;
  const uint64_t want = rows.nhigh + (units + kThreads / 32 - 1) / (kThreads / 32);
  const int grid = (int)std::min<uint64_t>(std::max<uint64_t>(want, 1), (uint64_t)*per_sm * sms);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeCooperative;
  at.val.cooperative = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_persist<MODE>, a, rows);
}

cudaError_t launch_persist(const SolveArgs& a, const GraphDev& g, int mode, int sms, int per_sm[4], cudaStream_t s) {
  const PersistRows rows = {g.cls_begin[MID], g.cls_begin[HIGH] - g.cls_begin[MID], g.cls_begin[HIGH],
                            g.cls_begin[NCLS] - g.cls_begin[HIGH]};
  switch (mode) {
    case PRX_DYNAMIC_TRAVERSAL: return persist_t<PRX_DYNAMIC_TRAVERSAL>(a, rows, sms, &per_sm[1], s);
    case PRX_DYNAMIC_FRONTIER: return persist_t<PRX_DYNAMIC_FRONTIER>(a, rows, sms, &per_sm[2], s);
    case PRX_PRUNE_DYNAMIC_FRONTIER: return persist_t<PRX_PRUNE_DYNAMIC_FRONTIER>(a, rows, sms, &per_sm[3], s);
    default: return persist_t<PRX_STATIC>(a, rows, sms, &per_sm[0], s);
  }
}

}  // namespace prx
