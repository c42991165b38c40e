// Correctly rounded FP64 addition of non-negative doubles in integer
// operations only (host and device).
//
// GB300 executes FP64 at 2 lanes per SM per clock, so a warp-wide DADD holds
// an SM's FP64 pipe for 16 cycles (20 measured) while its integer pipes run 64
// lanes per clock.  The sweeps add one contribution per edge in the
// reference's order; moving part of the adds to the integer pipes keeps the
// order and the bits (IEEE 754 addition is a function of its two operands)
// and spreads the work over both.
//
// The method is the guard / round / sticky adder of IEEE 754 arithmetic
// (D. Goldberg, "What every computer scientist should know about
// floating-point arithmetic", ACM Computing Surveys 23(1), 1991, section 1.4):
// align the smaller significand to the larger one keeping three extra bits,
// the lowest the OR of every bit shifted past it; add; on a carry shift one
// more bit into the sticky one; round to nearest, ties to even.  For operands
// of one sign nothing cancels, so no normalisation beyond that carry is
// needed.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define PRX_HD __host__ __device__ __forceinline__
#else
#define PRX_HD inline
#endif

namespace prx {

// add_nonneg_bits takes operands whose high words are below this: sign clear
// and biased exponent below 2000, i.e. values below 2^977.  A sum of up to
// 2^32 such terms stays below 2^1009, so no addition along a row overflows.
constexpr uint32_t kSoftAddHiLimit = 2000u << 20;

// Bits of RN(x + y) for the bit patterns x, y of two doubles whose high words
// are below kSoftAddHiLimit (zeros and subnormals included): the method in one
// function, as the host test checks it.  The kernels take soft_add below.
PRX_HD uint64_t add_nonneg_bits(uint64_t x, uint64_t y) {
  // non-negative doubles order as their bit patterns
  const uint64_t h = x > y ? x : y, l = x > y ? y : x;
  const uint32_t eh = (uint32_t)(h >> 52), el = (uint32_t)(l >> 52);
  // a subnormal has exponent 1 and no hidden bit
  const uint32_t Eh = eh > 1u ? eh : 1u, El = el > 1u ? el : 1u;
  // significands: the exponent field replaced by the hidden bit (1 if the
  // field was non-zero), then three guard bits below
  const uint64_t mh = (h - ((uint64_t)(Eh - 1u) << 52)) << 3;
  const uint64_t ml = (l - ((uint64_t)(El - 1u) << 52)) << 3;
  const uint32_t d = Eh - El;
  const uint32_t k = d < 63u ? d : 63u;  // ml < 2^56: a shift of 56 or more leaves only the sticky bit
  const uint64_t al = ml >> k;
  uint64_t s = mh + (al | (uint64_t)((al << k) != ml));  // < 2^57
  const uint32_t c = (uint32_t)(s >> 56);                // carry out of the significand
  s = (s >> c) | (s & (uint64_t)c);
  const uint64_t r = s >> 3;
  // round up when the three extra bits exceed one half, or equal it and r is odd
  const uint64_t q = r + ((((uint32_t)s & 7u) + ((uint32_t)r & 1u) + 3u) >> 3);
  // q carries the hidden bit at 52 (a rounding carry into bit 53 moves to the
  // next binade), so adding it to the exponent field minus one is the encoding
  return ((uint64_t)(Eh + c - 1u) << 52) + q;
}

// The same sum in fewer operations for a running sum kept unpacked: value
// (hi:lo) * 2^(e - 1075), hidden bit at bit 52.  The smaller significand is
// shifted right by the exponent difference with every bit kept (64 below the
// larger one's last place), so no sticky bit has to be formed: the fraction F
// below the sum's last place is exact, and the sum is rounded up when
// F > 1/2, or F = 1/2 and the last place is odd -- "odd" goes into F's lowest
// bit, which is always 0, and one comparison decides both.  A shift of 63 or
// more leaves F below 1/2 whatever the operand was, so an addend that is zero
// or subnormal needs no case of its own as long as the running sum is at
// least 2^-895 (kSoftMinHi).
//
// Measured on GB300 (cycles per warp-wide addition and SM, throughput /
// latency): DADD 20 / 65, add_nonneg_bits 22 / 110, soft_add 14 / 79, and 10
// when half of the additions are DADDs.
struct SoftAcc {
  uint32_t e, hi, lo;
};

// soft_add takes a running sum whose high word is in [kSoftMinHi,
// kSoftAddHiLimit) and addends below kSoftAddHiLimit.  Sums of up to 2^32
// such terms stay in the range.
constexpr uint32_t kSoftMinHi = 128u << 20;

PRX_HD SoftAcc soft_unpack(uint64_t x) {
  const uint32_t h = (uint32_t)(x >> 32);
  return {h >> 20, (h & 0xfffffu) | 0x100000u, (uint32_t)x};
}
PRX_HD uint64_t soft_pack(const SoftAcc& a) {
  return ((uint64_t)((a.e << 20) + (a.hi & 0xfffffu)) << 32) | a.lo;
}

PRX_HD SoftAcc soft_add(const SoftAcc& a, uint64_t x) {
  const uint32_t xh = (uint32_t)(x >> 32), xl = (uint32_t)x;
  const uint32_t ex = xh >> 20, mh = (xh & 0xfffffu) | 0x100000u;
  const bool swap = ex > a.e;
  const uint32_t bh = swap ? mh : a.hi, bl = swap ? xl : a.lo, sh = swap ? a.hi : mh, sl = swap ? a.lo : xl;
  const uint32_t E = swap ? ex : a.e, diff = E - (swap ? a.e : ex);
  const uint32_t d = diff < 63u ? diff : 63u;
  const uint64_t s = ((uint64_t)sh << 32) | sl;
  uint64_t down, lost;  // s >> d, and the bits shifted out at the top of 64
#if defined(__CUDA_ARCH__)
  asm("shr.u64 %0, %1, %2;" : "=l"(down) : "l"(s), "r"(d));
  asm("shl.b64 %0, %1, %2;" : "=l"(lost) : "l"(s), "r"(64u - d));  // a shift of 64 gives 0
#else
  down = s >> d;
  lost = d ? s << (64u - d) : 0;
#endif
  const uint64_t S = (((uint64_t)bh << 32) | bl) + down;
  const uint32_t c = (uint32_t)(S >> 53);  // carry: the sum's last place is one bit up
  SoftAcc o;
#if defined(__CUDA_ARCH__)
  const uint32_t Sl = (uint32_t)S, Sh = (uint32_t)(S >> 32), Ll = (uint32_t)lost, Lh = (uint32_t)(lost >> 32);
  const uint32_t Hl = __funnelshift_r(Sl, Sh, c), Hh = Sh >> c;
  const uint32_t Fh = __funnelshift_r(Lh, Sl, c), Fl = __funnelshift_r(Ll, Lh, c) | (Hl & 1u);
  uint32_t rl, rh;
  asm("{\n\t.reg .u32 x;\n\t"
      "add.cc.u32 x, %2, 0xffffffff;\n\taddc.cc.u32 x, %3, 0x7fffffff;\n\t"  // carries when F > 2^63
      "addc.cc.u32 %0, %4, 0;\n\taddc.u32 %1, %5, 0;\n\t}"
      : "=r"(rl), "=r"(rh)
      : "r"(Fl), "r"(Fh), "r"(Hl), "r"(Hh));
#else
  const uint64_t H = S >> c, F = (c ? (S << 63) | (lost >> 1) : lost) | (H & 1u);
  const uint64_t r = H + (F > 0x8000000000000000ull ? 1u : 0u);
  const uint32_t rl = (uint32_t)r, rh = (uint32_t)(r >> 32);
#endif
  const uint32_t c2 = rh >> 21;  // the rounding reached the next binade: all other bits are 0
  o.e = E + c + c2;
  o.hi = rh >> c2;
  o.lo = rl;
  return o;
}

// a / d correctly rounded in integer operations, for a positive normal a
// (high word ah) and an integer d >= 1 with R = quot_table_entry(d), the
// 64-bit normalised reciprocal floor(2^(64+b) / d), b = floor(log2 d): the
// product of the left-justified significand and R, cut to 64 bits, lies
// within 4 units of the exact quotient below it (one for R's floor, one for
// the cut, doubled by the normalisation), and an exact quotient of a 53-bit
// by a 32-bit number is never halfway between two 53-bit numbers; so the
// rounding is decided unless the estimate's 11 low bits are in the three
// units below one half.  *undecided is set there (0.15% of quotients), and
// the caller divides otherwise.  Measured: 11.5 cycles per warp and SM
// against 64 for the three FP64 operations of div_count and its conversion.
constexpr uint32_t kQuotMinHi = 64u << 20, kQuotHiRange = 1900u << 20;  // ah in [min, min + range)

PRX_HD uint64_t quot_bits(uint64_t a, uint32_t d, uint64_t R, bool* undecided) {
  const uint32_t ah = (uint32_t)(a >> 32);
  const uint64_t A = (a << 11) | 0x8000000000000000ull;
#if defined(__CUDA_ARCH__)
  const uint64_t q = __umul64hi(A, R);  // in [2^62 - 1, 2^64)
  const uint32_t b = 31u - (uint32_t)__clz((int)d);
#else
  const uint64_t q = (uint64_t)(((unsigned __int128)A * R) >> 64);
  const uint32_t b = 31u - (uint32_t)__builtin_clz(d);
#endif
  const uint32_t s = (uint32_t)(q >> 63) ^ 1u;
  const uint64_t Q = q << s;
  *undecided = ((uint32_t)Q & 0x7ffu) - 0x3fdu < 3u;
  const uint64_t m = (Q >> 11) + (((uint32_t)Q >> 10) & 1u);
  return ((uint64_t)((ah >> 20) - b - s - 1u) << 52) + m;
}

PRX_HD uint64_t quot_table_entry(uint32_t d) {  // d >= 1
#if defined(__CUDA_ARCH__)
  const uint32_t b = 31u - (uint32_t)__clz((int)d);
#else
  const uint32_t b = 31u - (uint32_t)__builtin_clz(d);
#endif
  const uint64_t top = 1ull << (32 + b);
  const uint64_t hi = top / d;                      // 2^64 for a power of two: one less
  if (hi >> 32) return ~0ull;
  return (hi << 32) + ((top - hi * d) << 32) / d;
}

}  // namespace prx
