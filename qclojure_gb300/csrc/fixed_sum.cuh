// Sums of doubles in fixed point on the integer pipes.
//
// The reductions (Pauli strings, outcome probabilities) compensate every addition, and a TwoSum
// is seven instructions on the FP64 pipe, of which this part has two lanes per SM and clock: an
// FP64 instruction costs as much as 32 to 64 integer ones. Up to 4096 values of magnitude below
// 2^(E - 1022), E the biased exponent of the largest, are added exactly instead, as two integers
// each:
//   v = h 2^(E - 1063) + l 2^(E - 1111),  |h| < 2^41, |l| < 2^48,
// l cut off below its unit (2^-88 of the largest value; nothing is cut off of values above
// 2^-36 of it). Sums of h stay within 2^53 and convert exactly, sums of l within 2^60. One TwoSum
// takes the sum of a whole group, so the total is at least as accurate as one with a TwoSum per
// value (tests/test_fixed_sum.py), whatever the order or the signs.
//
// Host and device: the CPU test compiles this header with a host compiler.
#pragma once

#include "quant.cuh"

// v << r, 0 from r = 64 on
QG_QHD uint64_t qg_shl64(uint64_t v, unsigned r) {
#if defined(__CUDA_ARCH__)
  uint64_t o;
  asm("shl.b64 %0, %1, %2;" : "=l"(o) : "l"(v), "r"(r));
  return o;
#else
  return r > 63u ? 0ull : v << r;
#endif
}

// Grows with the magnitude of v; the largest key of a group gives its exponent (at least 37,
// where the unit of l is the smallest subnormal; 2047: an infinity or NaN is among the values).
QG_QHD uint32_t qg_fix_key(double v) { return (uint32_t)(qg_bits_of(v) >> 32) & 0x7FFFFFFFu; }
QG_QHD int qg_fix_exponent(uint32_t key) {
  const int e = (int)(key >> 20);
  return e < 37 ? 37 : e;
}

struct qg_fixed {
  int64_t h, l;
};
// v (negated where flip is 1) in the units of exponent E
QG_QHD qg_fixed qg_fix(double v, int E, uint32_t flip) {
  const uint64_t b = qg_bits_of(v);
  const int e = (int)((b >> 52) & 0x7FF);
  const uint64_t m = (b & 0xFFFFFFFFFFFFFull) | (e ? 1ull << 52 : 0ull);  // |v| = m 2^(max(e, 1) - 1075)
  const unsigned d = (unsigned)(E - (e ? e : 1));
  const uint64_t h = qg_shr64(m, d + 12u);
  // (m 2^(36 - d)) mod 2^48: one of the shifts has a count of 64 and more
  const uint64_t l = (qg_shl64(m, 36u - d) | qg_shr64(m, d - 36u)) & 0xFFFFFFFFFFFFull;
  const uint64_t s = 0ull - ((b >> 63) ^ (uint64_t)flip);
  return qg_fixed{(int64_t)((h ^ s) - s), (int64_t)((l ^ s) - s)};
}

// 2^(p - 1023) for p from -51 on
QG_QHD double qg_fix_unit(int p) { return qg_double_of(p >= 1 ? (uint64_t)p << 52 : 1ull << (p + 51)); }
// The value of a sum: hi + lo (NaN where the group holds an infinity or NaN, as a TwoSum gives)
QG_QHD double qg_fix_hi(int64_t h, int E) {
  return E == 0x7FF ? qg_double_of(0x7FF8000000000000ull) : (double)h * qg_fix_unit(E - 40);
}
QG_QHD double qg_fix_lo(int64_t l, int E) { return (double)l * qg_fix_unit(E - 88); }
