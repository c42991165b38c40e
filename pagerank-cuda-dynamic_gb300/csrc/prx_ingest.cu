// prx_ingest.cu -- both CSRs of an edge list, built on the device.
//
// What the reference assembles on the host (readTemporalOmpW, inc/snap.hxx:
// 158-166, addSelfLoopsOmp, inc/selfLoop.hxx:60-66, transposeWithDegreeOmp,
// inc/transpose.hxx:110-134): rows ascending, duplicates merged, a self-loop on
// every vertex when asked for, the transpose and the out-degrees.
//
// A row's order is all that is wanted, so nothing sorts the whole list.  The
// out-rows, and from the same list read the other way round the in-rows, are
//   1. counted and the counts scanned; the atomic that counts an entry gives
//      its place in the row, in any order,
//   2. filled,
//   3. sorted where they lie and their duplicates merged: rows of up to 8
//      entries by 8 lanes, up to 256 in a warp's registers, up to 16384 in a
//      block's shared memory, longer ones together by the radix sort on
//      (row, id),
//   4. closed up, when there were duplicates.
// What bounds it: 1 one random atomic an entry and CSR, 2 one random 4-byte
// write, 3 the sorts' instructions.  On a web-like list of 117M edges (3M
// vertices, in row order; all in ms): 1 1.1, 2 0.4 for the out-rows and 2.2 for
// the in-rows (their targets' sectors come and go 4 bytes at a time; grouping
// the entries by windows that stay in L2 first cost what it saved), 3 0.9 and
// 0.6, the radix sort of the rows that need it 0.9, 4 0.4.  Radix sorts of all
// keys took 11.9 in nine passes, the whole build 12.0 then and 8.3 now.
#include <algorithm>
#include "prx_ctx.h"
#include "prx_device.cuh"

namespace prx {

constexpr uint32_t kWarpSort = 256;     // longest row sorted in a warp's registers
constexpr uint32_t kBlockSort = 16384;  // longest row sorted in shared memory (64 KB)
constexpr uint32_t kSmallSort = 1024;   // ... by a block of 128 threads, the rest by 512
constexpr uint32_t kNoId = 0xffffffffu; // above every vertex id

// Rows left to a small block (mid), to a block (list) and to the radix sort
// (huge, huge_len).
struct LongRows {
  uint32_t* mid;
  uint32_t* list;
  uint32_t* huge;
  uint32_t* huge_len;
  uint32_t* count;  // [0] mid, [1] list, [2] huge, [3] huge rows' entries, [4] an id was out of range
};

// cnt[at] += 1 for the lanes of a full warp that have a row (at != kNoId), and
// the lane's own place among its row's.  One atomic per run of equal rows (lists
// in row order), or per distinct row once a row that two lanes are asked for
// came back in three runs (a hub): one counter takes an atomic every 0.65 ns.
// Matching every warp took 346 us where this takes 317 (17M entries, both ways);
// asking anew each time took 1515 us of 20M entries whose largest row had a sixth
// of them, and hubs, kept over the warp's entries, takes 713.
__device__ __forceinline__ uint32_t add_one(uint32_t* cnt, uint32_t at, bool& hubs) {
  const uint32_t lane = lane_id(), upto = 0xffffffffu >> (31 - lane);
  const uint32_t before = __shfl_up_sync(0xffffffffu, at, 1);
  const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || at != before);
  const unsigned hub0 = __ballot_sync(0xffffffffu, at == __shfl_sync(0xffffffffu, at, 0)) & heads;
  const unsigned hub1 = __ballot_sync(0xffffffffu, at == __shfl_sync(0xffffffffu, at, 16)) & heads;
  unsigned same;
  uint32_t leader;
  hubs = hubs || __popc(hub0) > 2 || __popc(hub1) > 2;
  if (hubs) {
    same = __match_any_sync(0xffffffffu, at);
    leader = __ffs(same) - 1;
  } else {
    leader = 31 - __clz(heads & upto);
    const unsigned later = heads & ~upto;  // the runs after this lane's
    same = (later ? (1u << (__ffs(later) - 1)) - 1u : 0xffffffffu) & ~((1u << leader) - 1u);
  }
  uint32_t base = 0;
  if (lane == leader && at != kNoId) base = atomicAdd(cnt + at, (uint32_t)__popc(same));
  return __shfl_sync(0xffffffffu, base, leader) + __popc(same & (upto >> 1));
}

// Where row v's counter lies among 2^bits of them; bits 0: at v.  Hubs have
// neighbouring ids, and a 128-byte line takes an atomic every 0.65 ns: with the
// counters spread over all lines, 17M entries of a 2^20-vertex RMAT list are
// counted in 346 us instead of 558.  Not past 2^21 rows: such counters don't
// stay in L2 whole, and a list with locality (a 9M-vertex grid) took 1.3 ms more.
__device__ __forceinline__ uint32_t counter_of(uint32_t v, int bits) {
  return bits ? (v * 0x9e3779b1u) & ((1u << bits) - 1u) : v;
}

// Entries per out-row and in-row (both preset to the self-loops), and each
// entry's places in its two rows.
__global__ void __launch_bounds__(256) k_ing_count(const uint32_t* __restrict__ u, const uint32_t* __restrict__ v,
                                                   uint32_t count, uint32_t n, int bits,
                                                   uint32_t* __restrict__ out, uint32_t* __restrict__ in, uint32_t* __restrict__ at_out,
                                                   uint32_t* __restrict__ at_in, uint32_t* __restrict__ bad,
                                                   const uint32_t* __restrict__ heavy, uint32_t least) {
  if (heavy && *heavy >= least) return;  // radix keys instead
  const uint32_t step = gridDim.x * blockDim.x;
  bool out_hubs = false, in_hubs = false;
  for (uint32_t i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); i0 < count; i0 += step) {
    const uint32_t i = i0 + lane_id();
    const uint32_t a = i < count ? u[i] : kNoId, b = i < count ? v[i] : kNoId;
    const bool ok = a < n && b < n;
    if (i < count && !ok) *bad = 1u;
    const uint32_t p = add_one(out, ok ? counter_of(a, bits) : kNoId, out_hubs);
    const uint32_t q = add_one(in, ok ? counter_of(b, bits) : kNoId, in_hubs);
    if (ok) {
      at_out[i] = p;
      at_in[i] = q;
    }
  }
}

__global__ void k_ing_fill(uint32_t* __restrict__ x, uint64_t count, uint32_t value) {
  for (uint64_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) x[i] = value;
}

__global__ void k_ing_lengths(const uint32_t* __restrict__ out, const uint32_t* __restrict__ in, uint32_t n, int bits,
                              uint32_t* __restrict__ out_len, uint32_t* __restrict__ in_len) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += gridDim.x * blockDim.x) {
    const uint32_t at = counter_of(v, bits);
    out_len[v] = v < n ? out[at] : 0u;
    in_len[v] = v < n ? in[at] : 0u;
  }
}

// A self-loop takes its row's first place.
__global__ void k_ing_loops(const uint32_t* __restrict__ off, uint32_t n, uint32_t* __restrict__ edg) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) edg[off[v]] = v;
}

// Entry (u, v) to its place in row u.
__global__ void __launch_bounds__(256) k_ing_place(const uint32_t* __restrict__ u, const uint32_t* __restrict__ v,
                                                   const uint32_t* __restrict__ at, uint32_t count, uint32_t n,
                                                   const uint32_t* __restrict__ off, uint32_t* __restrict__ edg) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const uint32_t a = u[i], b = v[i], k = at[i];
    if (a < n && b < n) edg[(uint32_t)(off[a] + k)] = b;
  }
}

// ---- row sorts -----------------------------------------------------------------
// Steps K0 .. 32 E of the ascending bitonic sort of 32 E values, value
// 32 e + lane in x[e] of its lane; descending when down.
template <int E, uint32_t K0 = 2>
__device__ __forceinline__ void warp_sort(uint32_t x[E], bool down = false) {
  const uint32_t lane = lane_id();
#pragma unroll
  for (uint32_t k = K0; k <= 32u * E; k <<= 1) {
#pragma unroll
    for (uint32_t j = k >> 1; j; j >>= 1) {
      if (j >= 32) {
        const uint32_t je = j >> 5;
#pragma unroll
        for (uint32_t e = 0; e < (uint32_t)E; ++e)
          if (!(e & je)) {
            const bool up = (!((e << 5) & k)) != (k == 32u * E && down);
            const uint32_t a = x[e], b = x[e | je];
            x[e] = up ? min(a, b) : max(a, b);
            x[e | je] = up ? max(a, b) : min(a, b);
          }
      } else {
#pragma unroll
        for (uint32_t e = 0; e < (uint32_t)E; ++e) {
          const uint32_t y = __shfl_xor_sync(0xffffffffu, x[e], j);
          const bool up = (!(((e << 5) | lane) & k)) != (k == 32u * E && down), low = !(lane & j);
          x[e] = up == low ? min(x[e], y) : max(x[e], y);
        }
      }
    }
  }
}

// Sort one row of at most 32 E entries, merge its duplicates and write the
// length that is left.
template <int E>
__device__ __forceinline__ void sort_row(uint32_t* __restrict__ row, uint32_t len, uint32_t* __restrict__ ulen) {
  const uint32_t lane = lane_id();
  uint32_t x[E];
#pragma unroll
  for (int e = 0; e < E; ++e) x[e] = 32u * e + lane < len ? row[32 * e + lane] : kNoId;
  warp_sort<E>(x);
  uint32_t kept = 0, last = kNoId;  // last: the value before this 32
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const uint32_t up = __shfl_up_sync(0xffffffffu, x[e], 1);
    const bool first = 32u * e + lane < len && x[e] != (lane ? up : last);
    last = __shfl_sync(0xffffffffu, x[e], 31);
    const unsigned mask = __ballot_sync(0xffffffffu, first);
    if (first) row[kept + __popc(mask & ((1u << lane) - 1u))] = x[e];
    kept += __popc(mask);
  }
  if (lane == 0) *ulen = kept;
}

// A warp takes four consecutive rows: side by side when none has more than 8
// entries, else one after the other.
__global__ void __launch_bounds__(256) k_ing_sort(const uint32_t* __restrict__ off, uint32_t n,
                                                  uint32_t* __restrict__ edg, uint32_t* __restrict__ ulen,
                                                  LongRows lr) {
  const uint32_t lane = lane_id();
  const uint32_t quads = (uint32_t)(((uint64_t)n + 3) / 4);
  for (uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < quads; q += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t v0 = 4 * q;
    const uint32_t bound = lane < 5 ? off[min(v0 + lane, n)] : 0u;          // rows past n are empty
    const uint32_t mine = __shfl_down_sync(0xffffffffu, bound, 1) - bound;  // lanes 0 .. 3: row lengths
    const uint32_t longest = __reduce_max_sync(0xffffffffu, lane < 4 ? mine : 0u);
    if (longest <= 8) {
      const uint32_t g = lane >> 3, i = lane & 7u;
      const uint32_t s = __shfl_sync(0xffffffffu, bound, g), len = __shfl_sync(0xffffffffu, mine, g);
      uint32_t x = i < len ? edg[s + i] : kNoId;
#pragma unroll
      for (uint32_t k = 2; k <= 8; k <<= 1)
#pragma unroll
        for (uint32_t j = k >> 1; j; j >>= 1) {
          const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
          x = (!(i & k) == !(i & j)) ? min(x, y) : max(x, y);
        }
      const uint32_t up = __shfl_up_sync(0xffffffffu, x, 1);
      const bool first = i < len && (i == 0 || x != up);
      const unsigned mask = (__ballot_sync(0xffffffffu, first) >> (8 * g)) & 0xffu;
      if (first) edg[s + __popc(mask & ((1u << i) - 1u))] = x;
      if (i == 0 && v0 + g < n) ulen[v0 + g] = __popc(mask);
      continue;
    }
    for (uint32_t r = 0; r < 4; ++r) {
      const uint32_t v = v0 + r;
      if (v >= n) break;
      const uint32_t s = __shfl_sync(0xffffffffu, bound, r), len = __shfl_sync(0xffffffffu, mine, r);
      if (len <= 32) sort_row<1>(edg + s, len, ulen + v);
      else if (len <= 64) sort_row<2>(edg + s, len, ulen + v);
      else if (len <= 128) sort_row<4>(edg + s, len, ulen + v);
      else if (len <= kWarpSort) sort_row<8>(edg + s, len, ulen + v);
      else if (lane == 0) {
        if (len <= kSmallSort) {
          lr.mid[atomicAdd(lr.count, 1u)] = v;
        } else if (len <= kBlockSort) {
          lr.list[atomicAdd(lr.count + 1, 1u)] = v;
        } else {
          const uint32_t at = atomicAdd(lr.count + 2, 1u);
          lr.huge[at] = v;
          lr.huge_len[at] = len;
          atomicAdd(lr.count + 3, len);
        }
      }
    }
  }
}

// The listed rows, a block of T threads each, in shared memory: 256 entries at
// a time in a warp's registers, the bitonic steps wider than that between them.
template <int T>
__global__ void __launch_bounds__(T) k_ing_sort_block(const uint32_t* __restrict__ off, uint32_t* __restrict__ edg,
                                                      uint32_t* __restrict__ ulen, const uint32_t* __restrict__ list,
                                                      const uint32_t* __restrict__ listed) {
  extern __shared__ uint32_t x[];
  constexpr uint32_t W = T / 32;
  __shared__ uint32_t part[32];
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  const uint32_t count = *listed;
  if (threadIdx.x < 32) part[threadIdx.x] = 0;
  for (uint32_t b = blockIdx.x; b < count; b += gridDim.x) {
    const uint32_t v = list[b];
    const uint32_t s = off[v], len = off[v + 1] - s;
    uint32_t P = 512;
    while (P < len) P <<= 1;
    uint32_t y[8];
    for (uint32_t c = warp; c < P / 256; c += W) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const uint32_t i = 256 * c + 32 * e + lane;
        y[e] = i < len ? edg[s + i] : kNoId;
      }
      warp_sort<8>(y, c & 1);
#pragma unroll
      for (int e = 0; e < 8; ++e) x[256 * c + 32 * e + lane] = y[e];
    }
    __syncthreads();
    for (uint32_t k = 512; k <= P; k <<= 1) {
      for (uint32_t j = k >> 1; j >= 256; j >>= 1) {
        for (uint32_t t = threadIdx.x; t < P / 2; t += T) {
          const uint32_t i = 2 * t - (t & (j - 1)), l = i | j;
          const uint32_t p = x[i], q = x[l];
          if ((p > q) == !(i & k)) {
            x[i] = q;
            x[l] = p;
          }
        }
        __syncthreads();
      }
      for (uint32_t c = warp; c < P / 256; c += W) {
#pragma unroll
        for (int e = 0; e < 8; ++e) y[e] = x[256 * c + 32 * e + lane];
        warp_sort<8, 256>(y, (256 * c) & k);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[256 * c + 32 * e + lane] = y[e];
      }
      __syncthreads();
    }
    uint32_t kept = 0;
    for (uint32_t base = 0; base < len; base += T) {
      const uint32_t i = base + threadIdx.x;
      const bool first = i < len && (i == 0 || x[i] != x[i - 1]);
      const unsigned mask = __ballot_sync(0xffffffffu, first);
      if (lane == 0) part[warp] = __popc(mask);
      __syncthreads();
      const uint32_t c = part[lane];
      const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? c : 0u);
      if (first) edg[s + kept + before + __popc(mask & ((1u << lane) - 1u))] = x[i];
      kept += __reduce_add_sync(0xffffffffu, c);
      __syncthreads();
    }
    if (threadIdx.x == 0) ulen[v] = kept;
  }
}

// ---- rows past a block's shared memory: all of them in one key list, huge row
// b's entries as b << vbits | id from base[b] on ------------------------------------------
__global__ void k_ing_huge_keys(const uint32_t* __restrict__ off, const uint32_t* __restrict__ edg, LongRows lr,
                                uint32_t rows, int vbits, const uint32_t* __restrict__ base,
                                unsigned long long* __restrict__ key) {
  const uint32_t sum = base[rows];
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < sum; i += gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = rows;  // base[lo] <= i < base[hi]
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (base[mid] <= i) lo = mid;
      else hi = mid;
    }
    key[i] = ((unsigned long long)lo << vbits) | edg[(uint32_t)(off[lr.huge[lo]] + (i - base[lo]))];
  }
}

__global__ void k_ing_huge_first(const unsigned long long* __restrict__ key, uint32_t sum,
                                 uint32_t* __restrict__ pos) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= sum; i += gridDim.x * blockDim.x)
    pos[i] = i < sum && (i == 0 || key[i] != key[i - 1]) ? 1u : 0u;
}

// pos: the scanned flags above; sum + 1 of them.
__global__ void k_ing_huge_rows(const uint32_t* __restrict__ off, uint32_t* __restrict__ edg,
                                uint32_t* __restrict__ ulen, LongRows lr, uint32_t rows, int vbits,
                                const uint32_t* __restrict__ base, const uint32_t* __restrict__ pos,
                                const unsigned long long* __restrict__ key) {
  const uint32_t sum = base[rows];
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < sum; i += gridDim.x * blockDim.x) {
    const unsigned long long k = key[i];
    const uint32_t r = (uint32_t)(k >> vbits), v = lr.huge[r], from = base[r];
    if (pos[i + 1] != pos[i]) edg[(uint32_t)(off[v] + (pos[i] - pos[from]))] = (uint32_t)(k & ((1ull << vbits) - 1));
    if (i == from) ulen[v] = pos[base[r + 1]] - pos[from];
  }
}

// ---- closing up -------------------------------------------------------------------
// The unique entries of 32 rows per warp, spread over its lanes, from the
// places where the rows were sorted to the final CSR.  Long rows are the
// kernel below's: one of a million entries would keep its warp for long.
__global__ void __launch_bounds__(256) k_ing_close(const uint32_t* __restrict__ raw_off,
                                                   const uint32_t* __restrict__ raw, const uint32_t* __restrict__ off,
                                                   uint32_t n, uint32_t* __restrict__ edg) {
  const uint32_t lane = lane_id();
  const uint32_t words = (uint32_t)(((uint64_t)n + 31) >> 5);
  for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < words; w += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t v = (w << 5) | lane;
    uint32_t from = 0, to = 0, len = 0;
    if (v < n) {
      from = raw_off[v];
      to = off[v];
      if (raw_off[v + 1] - from <= kWarpSort) len = off[v + 1] - to;
    }
    uint32_t end = len;  // entries of the rows up to and with v
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= (uint32_t)o) end += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, end, 31);
    from -= end - len;  // entry t of row v: from + t
    to -= end - len;
    for (uint32_t t0 = 0; t0 < total; t0 += 32) {
      const uint32_t t = t0 + lane;
      uint32_t own = 0;  // the first row whose end exceeds t
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        const uint32_t y = __shfl_sync(0xffffffffu, end, own + o - 1);
        if (y <= t) own += o;
      }
      const uint32_t src = __shfl_sync(0xffffffffu, from, own), dst = __shfl_sync(0xffffffffu, to, own);
      if (t < total) edg[(uint32_t)(dst + t)] = raw[(uint32_t)(src + t)];
    }
  }
}

__global__ void __launch_bounds__(256) k_ing_close_long(const uint32_t* __restrict__ list, uint32_t count,
                                                        const uint32_t* __restrict__ raw_off,
                                                        const uint32_t* __restrict__ raw,
                                                        const uint32_t* __restrict__ off, uint32_t* __restrict__ edg) {
  for (uint32_t b = blockIdx.x; b < count; b += gridDim.x) {
    const uint32_t v = list[b], from = raw_off[v], to = off[v], len = off[v + 1] - to;
    for (uint32_t i = blockIdx.y * blockDim.x + threadIdx.x; i < len; i += gridDim.y * blockDim.x)
      edg[to + i] = raw[from + i];
  }
}

static int ing_grid(uint64_t threads, int sms) {
  const uint64_t b = (threads + 255) / 256;
  return (int)std::max<uint64_t>(1, std::min<uint64_t>(b, (uint64_t)sms * 16));
}

// Sort every row of edg (bounds off) and merge its duplicates, ulen[v] = the
// entries left.  Waits for the stream (found: LongRows::count).
static cudaError_t sort_rows(const uint32_t* off, uint32_t n, uint32_t* edg, uint32_t* ulen, const LongRows& lr,
                             uint32_t found[5], int sms, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(lr.count, 0, 4 * sizeof(uint32_t), s);
  if (e != cudaSuccess) return e;
  k_ing_sort<<<ing_grid((uint64_t)n * 8, sms), 256, 0, s>>>(off, n, edg, ulen, lr);
  e = cudaMemcpyAsync(found, lr.count, 5 * sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess || found[4]) return e;
  if (found[0])
    k_ing_sort_block<128><<<std::min<uint32_t>(found[0], 16u * sms), 128, kSmallSort * sizeof(uint32_t), s>>>(
        off, edg, ulen, lr.mid, lr.count);
  if (found[1]) {
    constexpr int smem = kBlockSort * sizeof(uint32_t);
    e = cudaFuncSetAttribute(k_ing_sort_block<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    k_ing_sort_block<512><<<std::min<uint32_t>(found[1], 3u * sms), 512, smem, s>>>(off, edg, ulen, lr.list,
                                                                                    lr.count + 1);
  }
  const uint32_t rows = found[2];
  if (rows) {
    const uint32_t sum = found[3];
    uint32_t *base = nullptr, *pos = nullptr, *hist = nullptr;
    unsigned long long *key = nullptr, *tmp = nullptr, *sorted = nullptr;
    e = graph_alloc(&base, sizeof(uint32_t) * ((size_t)rows + 1), s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(base, lr.huge_len, sizeof(uint32_t) * rows, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(base + rows, 0, sizeof(uint32_t), s);
    if (e == cudaSuccess) e = exclusive_scan_u32(base, rows + 1, s);
    if (e == cudaSuccess) e = graph_alloc(&key, 8 * ((size_t)sum + 2), s);
    if (e == cudaSuccess) e = graph_alloc(&tmp, 8 * ((size_t)sum + 2), s);
    if (e == cudaSuccess) e = graph_alloc(&pos, sizeof(uint32_t) * ((size_t)sum + 1), s);
    if (e == cudaSuccess) e = graph_alloc(&hist, sizeof(uint32_t) * radix_hist_words(sum), s);
    if (e == cudaSuccess) {
      int vbits = 1, rbits = 0;
      while (vbits < 32 && (1ull << vbits) < n) ++vbits;
      while ((1ull << rbits) < rows) ++rbits;
      const int grid = ing_grid((uint64_t)sum + 1, sms);
      k_ing_huge_keys<<<grid, 256, 0, s>>>(off, edg, lr, rows, vbits, base, key);
      e = radix_sort_u64(key, tmp, sum, 0, vbits + rbits, hist, sms, s, &sorted);
      if (e == cudaSuccess) {
        k_ing_huge_first<<<grid, 256, 0, s>>>(sorted, sum, pos);
        e = exclusive_scan_u32(pos, sum + 1, s);
        k_ing_huge_rows<<<grid, 256, 0, s>>>(off, edg, ulen, lr, rows, vbits, base, pos, sorted);
      }
    }
    for (void* p : {(void*)base, (void*)key, (void*)tmp, (void*)pos, (void*)hist})
      if (p) cudaFreeAsync(p, s);
  }
  return e == cudaSuccess ? cudaGetLastError() : e;
}

// One CSR of the list's entries u -> v: raw_off holds the rows' lengths with
// duplicates (scanned here); off receives the row starts, *edg the entries; of
// the out-rows (deg not null) deg the lengths and *m the number of entries.
static cudaError_t build_csr(uint32_t* raw_off, const uint32_t* u, const uint32_t* v, uint32_t count, uint32_t n,
                             bool loops, const uint32_t* at, const LongRows& lr, uint32_t* off, uint32_t* deg,
                             uint32_t** edg, uint32_t* m, bool* bad_id, int sms, cudaStream_t s) {
  const uint32_t total = count + (loops ? n : 0);
  uint32_t* raw = nullptr;
  cudaError_t e = graph_alloc(&raw, sizeof(uint32_t) * edge_slots(total), s);
  if (e != cudaSuccess) return e;
  uint32_t found[5] = {};
  e = exclusive_scan_u32(raw_off, n + 1, s);
  if (e == cudaSuccess) {
    if (loops) k_ing_loops<<<ing_grid(n, sms), 256, 0, s>>>(raw_off, n, raw);
    if (count) k_ing_place<<<ing_grid(count, sms), 256, 0, s>>>(u, v, at, count, n, raw_off, raw);
    e = sort_rows(raw_off, n, raw, off, lr, found, sms, s);
  }
  *bad_id = found[4] != 0;
  if (e == cudaSuccess && !*bad_id) {
    if (deg) e = cudaMemcpyAsync(deg, off, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(off + n, 0, sizeof(uint32_t), s);
    if (e == cudaSuccess) e = exclusive_scan_u32(off, n + 1, s);
    if (deg) {  // the in-rows have as many
      if (e == cudaSuccess) e = cudaMemcpyAsync(m, off + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    if (e == cudaSuccess && *m == total) {  // no duplicates: closed up already
      *edg = raw;
      return cudaSuccess;
    }
    if (e == cudaSuccess) e = graph_alloc(edg, sizeof(uint32_t) * edge_slots(*m), s);
    if (e == cudaSuccess) {
      k_ing_close<<<ing_grid(n, sms), 256, 0, s>>>(raw_off, raw, off, n, *edg);
      auto close_long = [&](const uint32_t* list, uint32_t rows, uint32_t split) {
        if (rows)
          k_ing_close_long<<<dim3(std::min<uint32_t>(rows, 16u * sms), split), 256, 0, s>>>(list, rows, raw_off, raw,
                                                                                           off, *edg);
      };
      close_long(lr.mid, found[0], 1);
      close_long(lr.list, found[1], 8);
      close_long(lr.huge, found[2], 32);
      e = cudaGetLastError();
    }
  }
  cudaFreeAsync(raw, s);
  return e;
}

cudaError_t build_csr_pair(GraphDev& g, const uint32_t* u, const uint32_t* v, uint32_t count, bool self_loops,
                           bool* bad_id, int sms, cudaStream_t s, HeavyRows* heavy) {
  const uint32_t n = g.n;
  const uint32_t total = count + (self_loops ? n : 0);
  *bad_id = false;
  const size_t rows = (size_t)n + 1;
  const size_t nm = total / (kWarpSort + 1) + 1, nl = total / (kSmallSort + 1) + 1,
               nh = total / (kBlockSort + 1) + 1;  // rows as long as that, at most
  int bits = 0;
  if (n <= 1u << 21)
    for (bits = 18; (1u << bits) < n;) ++bits;
  const size_t counters = bits ? (size_t)1 << bits : rows;
  uint32_t *ws = nullptr, m = 0;
  auto alloc = [&](uint32_t** p, size_t words) { return graph_alloc(p, sizeof(uint32_t) * (words ? words : 1), s); };
  cudaError_t e = alloc(&ws, 2 * counters + 2 * rows + 2 * (size_t)count + nm + nl + 2 * nh + 5);
  if (e == cudaSuccess) e = alloc(&g.xoff, rows);
  if (e == cudaSuccess) e = alloc(&g.xtoff, rows);
  if (e == cudaSuccess) e = alloc(&g.xtdat, n);
  if (e == cudaSuccess) {
    uint32_t *cnt = ws, *out = cnt + 2 * counters, *in = out + rows, *at_out = in + rows, *at_in = at_out + count, *lists = at_in + count;
    uint32_t* rest = lists + 5;
    const LongRows lr{rest, rest + nm, rest + nm + nl, rest + nm + nl + nh, lists};
    e = cudaMemsetAsync(lists, 0, 5 * sizeof(uint32_t), s);
    k_ing_fill<<<ing_grid(2 * counters, sms), 256, 0, s>>>(cnt, 2 * counters, self_loops ? 1u : 0u);
    if (count)
      k_ing_count<<<ing_grid(count, sms), 256, 0, s>>>(u, v, count, n, bits, cnt, cnt + counters, at_out, at_in,
                                                        lr.count + 4, heavy ? heavy->share : nullptr,
                                                        heavy ? heavy->least : 0u);
    k_ing_lengths<<<ing_grid(rows, sms), 256, 0, s>>>(cnt, cnt + counters, n, bits, out, in);
    if (e == cudaSuccess && heavy && heavy->share) {
      e = cudaEventSynchronize(heavy->ready);  // (while the entries are counted)
      heavy->found = e == cudaSuccess && *heavy->host >= heavy->least;
    }
    if (heavy && heavy->found) {
      graph_free({ws, g.xoff, g.xtoff, g.xtdat});
      g.xoff = g.xtoff = g.xtdat = nullptr;
      return e;
    }
    if (e == cudaSuccess)
      e = build_csr(out, u, v, count, n, self_loops, at_out, lr, g.xoff, g.xtdat, &g.xedg, &m, bad_id, sms, s);
    if (e == cudaSuccess && !*bad_id)
      e = build_csr(in, v, u, count, n, self_loops, at_in, lr, g.xtoff, nullptr, &g.xtedg, &m, bad_id, sms, s);
    g.m = g.m_cap = m;
  }
  if (ws) cudaFreeAsync(ws, s);
  return e == cudaSuccess ? cudaGetLastError() : e;
}

}  // namespace prx
