// Host check of prx::soft_add (a running sum kept unpacked) against the FPU's
// addition, and of prx::quot_bits against its division, on seeded operands in
// the ranges the kernels hand over.  Prints the mismatch count and exits
// non-zero on any mismatch.
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "prx_softadd.h"

static uint64_t bits_of(double a) {
  uint64_t u;
  memcpy(&u, &a, 8);
  return u;
}
static double from_bits(uint64_t u) {
  double a;
  memcpy(&a, &u, 8);
  return a;
}
static uint64_t seed = 99;
static uint64_t rnd() {  // splitmix64
  uint64_t z = (seed += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
static const uint64_t M52 = (1ull << 52) - 1;
static uint64_t mant() {
  switch (rnd() % 8) {
    case 0: return 0;
    case 1: return M52;
    case 2: return M52 - rnd() % 8;
    case 3: return rnd() % 8;
    case 4: return 1ull << (rnd() % 52);
    case 5: return (rnd() & M52) & ~((1ull << (rnd() % 52)) - 1);
    default: return rnd() & M52;
  }
}

int main() {
  long long sums = 0, quots = 0, undecided = 0, bad = 0;
  // sums: every exponent difference to +-70, ties and carries, addends zero and subnormal
  for (int row = 0; row < 400000; ++row) {
    uint64_t e = 128 + rnd() % 1800;
    uint64_t acc = (e << 52) | mant();
    prx::SoftAcc u = prx::soft_unpack(acc);
    for (int k = 0; k < 24; ++k) {
      const uint64_t ea = acc >> 52;
      uint64_t x;
      switch (rnd() % 8) {
        case 0: x = 0; break;
        case 1: x = rnd() & M52; break;  // subnormal
        default: {
          const long long ex = (long long)ea + 8 - (long long)(rnd() % 78);
          x = ex >= 1 && ex < 1990 ? ((uint64_t)ex << 52) | mant() : 0;
        }
      }
      if ((acc >> 32) >= prx::kSoftAddHiLimit) break;
      const volatile double a = from_bits(acc), b = from_bits(x);
      acc = bits_of(a + b);
      u = prx::soft_add(u, x);
      ++sums;
      if (prx::soft_pack(u) != acc) {
        if (bad++ < 10) printf("SUM %016llx + %016llx\n", (unsigned long long)bits_of(a), (unsigned long long)x);
        u = prx::soft_unpack(acc);
      }
    }
  }
  // an empty slot (+0) vanishes against a term on either side
  for (int i = 0; i < 1000; ++i) {
    const uint64_t x = ((128 + rnd() % 1800) << 52) | mant();
    bad += prx::soft_pack(prx::soft_add(prx::soft_unpack(0), x)) != x;
    const uint64_t two = prx::soft_pack(prx::soft_add(prx::soft_unpack(0), 0));
    bad += prx::soft_pack(prx::soft_add(prx::soft_unpack(two), x)) != x;
    bad += prx::soft_pack(prx::soft_add(prx::soft_unpack(x), two)) != x;
  }
  // quotients: small, power-of-two, large and extreme divisors
  for (int i = 0; i < 20000000; ++i) {
    uint32_t d;
    switch (rnd() % 5) {
      case 0: d = 1u << (rnd() % 32); break;
      case 1: d = (uint32_t)(0u - 1 - rnd() % 64); break;
      case 2: d = (uint32_t)rnd() | 1u; break;
      default: d = 1 + (uint32_t)(rnd() % 65535);
    }
    const uint64_t a = ((64 + rnd() % 1900) << 52) | mant();
    if ((uint32_t)(a >> 32) - prx::kQuotMinHi >= prx::kQuotHiRange) continue;
    bool open;
    const uint64_t q = prx::quot_bits(a, d, prx::quot_table_entry(d), &open);
    ++quots;
    undecided += open;
    const volatile double x = from_bits(a), y = (double)d;
    if (!open && q != bits_of(x / y)) {
      if (bad++ < 10) printf("QUOT %016llx / %u\n", (unsigned long long)a, d);
    }
  }
  printf("checked %lld sums, %lld quotients (%lld undecided), %lld mismatches\n", sums, quots, undecided, bad);
  return bad || undecided > quots / 200 ? 1 : 0;
}
