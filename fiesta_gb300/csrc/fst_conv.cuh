// fst_conv.cuh — FP64 <-> FP32 conversions on the integer pipe.
//
// GB300's FP64 unit also executes the F2F conversions, at the FP64 rate; these
// rebias the exponent and round the mantissa with integer operations instead.
// They are most of the integer work of the mixed path's equation of state (nine
// splits a cell), and the kernels that carry it are bound by instruction issue.
// Splitting with one rounding for both parts, the range tested once a cell and no
// redundant operations took the 256^3 species kernel with the equation of state
// (5 species) from 1511 to 1438 us and the primitive pass from 756 to 721 us.
#pragma once
#include "fst_fp64.cuh"

namespace fstm {

// high and low word (not fst64::bits_of: its opaque move costs these kernels 1.5 %)
struct words {
  uint32_t hi, lo;
};
FST_HD words words_of(double x) {
#if defined(__CUDA_ARCH__)
  return {(uint32_t)__double2hiint(x), (uint32_t)__double2loint(x)};
#else
  const uint64_t b = fst64::bits_of(x);
  return {(uint32_t)(b >> 32), (uint32_t)b};
#endif
}
// the high word of x without its sign: the range tests below are compares of it
FST_HD uint32_t abs_hi(double x) { return words_of(x).hi & 0x7FFFFFFFu; }
constexpr uint32_t F32_MIN_HI = 897u << 20;    // |x| >= 2^-126
constexpr uint32_t F32_OVER_HI = 1151u << 20;  // |x| >= 2^128, infinity or NaN

// The FP32 bits of x without its sign from the rounded bits of the normal range.
// Values outside it go to zero / infinity (no FP32 denormals); NaN stays NaN.
// Selects, no branch (zeros are common); the NaN test as words, which the compiler
// does not take for an FP64 compare.
FST_HD uint32_t clamp_bits(words u, uint32_t bits) {
  const uint32_t a = u.hi & 0x7FFFFFFFu;
  const bool nan = a >= 0x7FF00000u && ((a & 0xFFFFFu) | u.lo);
  bits = a < F32_MIN_HI ? 0u : bits;
  return a >= F32_OVER_HI ? (nan ? 0x7FC00000u : 0x7F800000u) : bits;
}

// The nearest FP32 value, mantissa ties away from zero.
FST_HD float d2f(double x) {
  const words u = words_of(x);
  // the low 9 exponent bits and 23 mantissa bits in one funnel shift, then the
  // exponent rebiased 1023 -> 127 (exact modulo 2^32 for the normal range) and the
  // dropped bits rounded; a carry rounds into the exponent.  (Rounding as in split,
  // in the 64-bit word, puts a carry chain before the shift: 560 us against 529 for
  // a step of the 24-case 2D ensemble.)
  uint32_t bits = fst64::shl_hi(u.lo, u.hi, 3) - (896u << 23);
  bits += (u.lo >> 28) & 1u;
  return fst64::float_of((u.hi & 0x80000000u) | clamp_bits(u, bits));
}

FST_HD double f2d(float x) {
  const uint32_t f = fst64::bits_of_f(x), a = f & 0x7FFFFFFFu;
  uint32_t hi = (a >> 3) + (896u << 20), lo = f << 29;  // exponent rebiased 127 -> 1023
  // inf / NaN: exponent 255 -> 2047; zero / FP32 denormal (selects, no branch)
  hi += a >= 0x7F800000u ? 896u << 20 : 0u;
  hi = a < 0x00800000u ? 0u : hi;
  lo = a < 0x00800000u ? 0u : lo;
  return fst64::of_bits((uint64_t)(hi | (f & 0x80000000u)) << 32 | lo);
}

struct f2p {
  float h, l;
};

// x as an FP32 pair: h = d2f(x), l = x - h (the 6 lowest bits of x truncated: 2^-46
// relative to x), no FP64 instruction.  One 64-bit add of 2^28 (with the exponent's
// rebias) rounds h and leaves w, the 29 dropped bits offset by half a unit of h: with
// E the unbiased exponent of x, x - h is (w - 2^28) 2^(E-52), whether h was rounded
// up or not.  It is formed exactly as F - 1.5 B with B = 2^(E-23) and
// F = B (1 + w / 2^29).  No low part when |x| < 2^-102.
// IN_RANGE: the caller has tested |x| < 2^128; otherwise such x give d2f(x) and no
// low part.
template <bool IN_RANGE = false>
FST_HD f2p split(double x) {
  const words u = words_of(x);
  const uint32_t a = u.hi & 0x7FFFFFFFu, sg = u.hi & 0x80000000u;
  const uint64_t b = ((uint64_t)u.hi << 32 | u.lo) + (0x10000000ull - (896ull << 52));
  const uint32_t w = (uint32_t)b;
  uint32_t bits = fst64::shl_hi(w, (uint32_t)(b >> 32), 3);
  bits = IN_RANGE ? (a < F32_MIN_HI ? 0u : bits) : clamp_bits(u, bits);
  const uint32_t B = sg | ((u.hi * 8u - (919u << 23)) & 0x7F800000u);  // FP32 exponent of 2^(E-23)
  const float F = fst64::float_of(B | ((w & 0x1FFFFFFFu) >> 6));
#if defined(__CUDA_ARCH__)
  const float r = __fmaf_rn(fst64::float_of(B), -1.5f, F);
#else
  const float r = fmaf(fst64::float_of(B), -1.5f, F);
#endif
  return {fst64::float_of(sg | bits), a < (921u << 20) || (!IN_RANGE && a >= F32_OVER_HI) ? 0.0f : r};
}

}  // namespace fstm
