// fst_fp64.cuh — IEEE double operations on the integer pipes.
//
// GB300 retires FP64 instructions at 2 lanes per clock and SM, 1/64 of its
// FP32 rate: one FP64 warp instruction holds a sub-partition's FP64 unit for
// 64 clocks, in which the scheduler can issue 64 others.  A division as the
// compiler emits it costs about 16 such slots.  The functions here give the
// same correctly rounded results from integer instructions (two per clock pair
// of pipes) while the FP64 unit works on something else.
//
// Everything is exact integer arithmetic after a reciprocal seed whose error is
// bounded in the comments; operands outside the stated range take the ordinary
// operator, so results equal the IEEE ones for every input.  The functions
// compile for the host too (the tests run them against the CPU's arithmetic).
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define FST_HD __host__ __device__ __forceinline__
#else
#define FST_HD inline
#endif

namespace fst64 {

FST_HD uint64_t bits_of(double x) {
#if defined(__CUDA_ARCH__)
  uint64_t b;  // an opaque move: integer tests on the bits stay integer tests
  asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
  return b;
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return b;
#endif
}
FST_HD double of_bits(uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)b);
#else
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}
FST_HD uint32_t mulhi_u32(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
// (hi:lo) << s, upper word, 0 < s < 32
FST_HD uint32_t shl_hi(uint32_t lo, uint32_t hi, int s) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(lo, hi, s);
#else
  return (hi << s) | (lo >> (32 - s));
#endif
}
// 1/f for f in [1, 2), relative error at most 2^-22.9
FST_HD float rcp_seed(float f) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  return r;
#elif defined(FST_RCP_SEED_HOST)
  return FST_RCP_SEED_HOST(f);
#else
  return 1.0f / f;
#endif
}
FST_HD float float_of(uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(b);
#else
  float f;
  memcpy(&f, &b, 4);
  return f;
#endif
}
FST_HD uint32_t bits_of_f(float f) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(f);
#else
  uint32_t b;
  memcpy(&b, &f, 4);
  return b;
#endif
}

// The rare operands' path, out of line: inlined, the operator would be predicated
// or run ahead of the test and take the FP64 unit's time for every operand.
#if defined(__CUDACC__)
__host__ __device__ __noinline__ static double div_any(double a, double b) { return a / b; }
__host__ __device__ __noinline__ static double mul_any(double a, double b) { return a * b; }
#else
inline double div_any(double a, double b) { return a / b; }
inline double mul_any(double a, double b) { return a * b; }
#endif

// R with R / 2^32 = 1/b' (1 - e), |e| < 2^-30, for the divisor mantissa b' = B
// / 2^52 in [1, 2), B its 53-bit integer (words bh with the implicit bit set,
// bl).  One Newton step in fixed point from the FP32 reciprocal:
//  - fb, b' truncated to 24 bits, is at most b' and above b' (1 - 2^-23), so the
//    seed is within (1 -+ 2^-21.9) / b'; times (1 - 2^-21), and not below 1/2, it
//    is below 1/b', by a relative e0 in (0, 2^-20.3), and below 1;
//  - bt R0 = 2^63 (1 - e0) up to b' truncated to 32 bits (2^-31); the step adds
//    R0 e0 with e0 cut to 2^-47, and leaves e0^2 < 2^-40, two truncations of at
//    most one unit (2^-31 each) and bt's 2^-31.
FST_HD uint32_t recip32(uint32_t bh, uint32_t bl) {
  const float fb = float_of((shl_hi(bl, bh, 3) & 0x7FFFFFu) | 0x3F800000u);
  const float r = fmaxf(rcp_seed(fb) * (1.0f - 1.0f / 2097152.0f), 0.5f);
  const uint32_t R0 = (bits_of_f(r) << 8) | 0x80000000u;
  const uint32_t bt = shl_hi(bl, bh, 11) | 0x80000000u;
  const uint64_t p = (uint64_t)bt * R0;
  const uint32_t e = ~(uint32_t)(p >> 16);  // e0 2^47, below 2^27
  return R0 + (mulhi_u32(R0, e) >> 15);
}

// floor(A 2^55 / B), A and B 53-bit mantissas (words ah, al and bh, bl, implicit
// bits set), R = recip32(bh, bl).  Two digits:
//  - q1 = A 2^31 / B to within 4 units (both factors carry 2^-30), lowered by 5:
//    the remainder A 2^31 - q1 B is in (0, 10 B), below 2^57;
//  - its quotient by B times 2^24, below 2^27.4, from the remainder's top 32
//    bits: in eighths of a unit the estimate is above the true value by less
//    than 1 and below it by less than 3, so (est - 1) / 8 is the floor or one
//    less, which the last remainder decides.
FST_HD uint64_t quot55(uint32_t ah, uint32_t al, uint32_t bh, uint32_t bl, uint32_t R) {
  const uint64_t B = ((uint64_t)bh << 32) | bl;
  const uint32_t at = shl_hi(al, ah, 11);
  const uint32_t q1 = mulhi_u32(at, R) - 5u;
  const uint64_t A31 = ((uint64_t)shl_hi(al, ah, 31) << 32) | (al << 31);
  const uint64_t r1 = A31 - ((uint64_t)q1 * bl + ((uint64_t)(q1 * bh) << 32));
  const uint32_t q2 = (mulhi_u32((uint32_t)(r1 >> 25), R) - 1u) >> 3;
  const uint64_t r2 = (r1 << 24) - ((uint64_t)q2 * bl + ((uint64_t)(q2 * bh) << 32));
  return ((uint64_t)q1 << 24) + q2 + (r2 >= B ? 1u : 0u);
}

// A divisor and its reciprocal, for several quotients by the same number.
struct Recip {
  uint32_t hi, lo, R;  // the words of the divisor, recip32 of its mantissa
};
FST_HD Recip recip_of(double b) {
  const uint64_t bb = bits_of(b);
  const uint32_t hi = (uint32_t)(bb >> 32), lo = (uint32_t)bb;
  return {hi, lo, recip32((hi & 0xFFFFFu) | 0x100000u, lo)};
}

// a / b, correctly rounded (to nearest, ties to even) for every input.
// Integer path: b normal, a normal or zero, and exponents at most 1000 apart, so
// that the quotient is normal; anything else takes the operator.  No quotient
// of two 53-bit mantissas lies half way between two 53-bit numbers (b times a
// 54-bit odd number has more than 53 significant bits), so rounding needs the
// quotient's integer bits alone.
// Measured on GB300, clocks of a sub-partition per warp: 129 (recip_of
// included) against the operator's 601, and hidden behind two FP64 operations.
// div_exact: operands for which div_core holds (a normal or zero, b normal, the quotient
// well inside the normal range).  Several quotients in one straight line, tested
// together afterwards, overlap: three in turn take one warp 800 clocks, three cores 335.
FST_HD bool div_exact(double a, const Recip& b) {
  const uint64_t ba = bits_of(a);
  const uint32_t ea = (uint32_t)(ba >> 52) & 0x7FFu, eb = (b.hi >> 20) & 0x7FFu;
  const uint32_t ex = (ba << 1) == 0 ? eb : ea;
  return !(ex - 1u >= 2046u || eb - 1u >= 2046u || ex + 1000u - eb > 2000u);
}
FST_HD double div_core(double a, const Recip& b) {
  const uint64_t ba = bits_of(a);
  const uint32_t ahi = (uint32_t)(ba >> 32), al = (uint32_t)ba;
  const uint32_t ea = (ahi >> 20) & 0x7FFu, eb = (b.hi >> 20) & 0x7FFu;
  const bool zero = (ba << 1) == 0;
  const uint32_t ex = zero ? eb : ea;
  const uint32_t ah = (ahi & 0xFFFFFu) | 0x100000u, bh = (b.hi & 0xFFFFFu) | 0x100000u;
  const uint64_t q = quot55(ah, al, bh, b.lo, b.R);
  const uint32_t t = (uint32_t)(q >> 55);  // 1: a' >= b', 56 bits
  const uint64_t m = (q + (2u << t)) >> (2 + t);
  const uint32_t hi = (uint32_t)(m >> 32) + ((ex - eb + 1021u + t) << 20);
  const uint32_t sg = (ahi ^ b.hi) & 0x80000000u;
  return of_bits(((uint64_t)((zero ? 0u : hi) | sg) << 32) | (zero ? 0u : (uint32_t)m));
}
FST_HD double div_by(double a, const Recip& b) {
  if (!div_exact(a, b)) return div_any(a, of_bits(((uint64_t)b.hi << 32) | b.lo));
  return div_core(a, b);
}
FST_HD double div_rn(double a, double b) { return div_by(a, recip_of(b)); }

// a 2^k, |k| <= 1000: an addition to the exponent where a and the result are
// normal (exact, as the multiplication is) or a is zero, else the
// multiplication by p = 2^k.
FST_HD double scale2(double a, int k, double p) {
  const uint64_t ba = bits_of(a);
  const uint32_t hi = (uint32_t)(ba >> 32);
  const uint32_t e = (hi >> 20) & 0x7FFu;
  const bool zero = (ba << 1) == 0;
  if (!zero && (e - 1u >= 2046u || e + (uint32_t)k - 1u >= 2046u)) return mul_any(a, p);
  return of_bits(((uint64_t)(hi + (zero ? 0u : (uint32_t)k << 20)) << 32) | (uint32_t)ba);
}
FST_HD double half(double a) { return scale2(a, -1, 0.5); }
FST_HD double twice(double a) { return scale2(a, 1, 2.0); }
FST_HD double eight(double a) { return scale2(a, 3, 8.0); }

#if defined(__CUDACC__)
// ---------------------------------------------------------------------------
// Sums and products as fused operations.  The unit takes a DFMA whose operands
// are three thread registers every 64 clocks a warp, but a DADD, DMUL or compare
// every 77 and a DFMA with an immediate, constant or uniform operand every 81 (GB300,
// every SM busy, independent chains).  x 1 + y and x y +
// (-0) round exactly as x + y and x y do, zeros' signs included.  lane_const
// keeps a constant in thread registers: n, a kernel argument that is never
// negative, makes it look different in every lane.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double lane_const(double c, int n) {
  uint32_t lane;
  asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
  return of_bits(bits_of(c) + ((uint64_t)(lane & (uint32_t)(n >> 31)) << 32));
}
struct Fused {
  double one, mzero;
  __device__ __forceinline__ explicit Fused(int n)
      : one(lane_const(1.0, n)), mzero(lane_const(-0.0, n)) {}
  __device__ __forceinline__ double add(double x, double y) const { return __fma_rn(x, one, y); }
  __device__ __forceinline__ double sub(double x, double y) const { return __fma_rn(-one, y, x); }
  __device__ __forceinline__ double mul(double x, double y) const { return __fma_rn(x, y, mzero); }
};
#endif

// ---------------------------------------------------------------------------
// Products.  Operands are normal or (where stated) zero and the caller's ranges
// keep every result normal, so that no test for special values is needed.
// Shifts of more than one word are written as multiplications by a power of two:
// they then run on the multiplier's pipe, which the logic leaves idle.
// ---------------------------------------------------------------------------
struct W2 {
  uint32_t h, l;
};
FST_HD W2 words(double x) {
  const uint64_t b = bits_of(x);
  return {(uint32_t)(b >> 32), (uint32_t)b};
}
// the upper word of the 53-bit mantissa of a normal number
FST_HD uint32_t mant_hi(uint32_t h) { return (h & 0xFFFFFu) | 0x100000u; }

// The double with mantissa M + round bit f's top, M = (m1, m0) in [2^52, 2^53],
// exponent field e20 >> 20 of the mantissa with its implicit bit, and sign:
// rounded up when f >= 2^31, and to even when f = 2^31 and nothing follows.  A
// mantissa that rounds up to 2^53 carries into the exponent.
FST_HD uint64_t round_join(uint32_t m1, uint32_t m0, uint32_t f, uint32_t rest, uint32_t e20,
                           uint32_t sign) {
  uint64_t r = (((uint64_t)(m1 + e20) << 32) | m0) + (f >> 31);
  if (((f ^ 0x80000000u) | rest) == 0) r &= ~1ull;
  return r | ((uint64_t)sign << 32);
}
// Rounds the 106-bit product of two 53-bit mantissas, words p3..p0 in [2^104,
// 2^106), e20: the exponent field (in place) of a product below 2^105.
FST_HD uint64_t round_product(uint64_t p32, uint32_t p1, uint32_t p0, uint32_t e20,
                              uint32_t sign) {
  const uint32_t p3 = (uint32_t)(p32 >> 32), p2 = (uint32_t)p32;
  const uint32_t n = p3 >> 9;        // 1: at least 2^105
  const uint32_t k = 4096u >> n;     // M = P >> (52 + n), from the words above p0
  const uint64_t t1 = (uint64_t)p1 * k;
  const uint64_t t2 = (uint64_t)p2 * k + (t1 >> 32);
  const uint32_t m1 = p3 * k + (uint32_t)(t2 >> 32);
  return round_join(m1, (uint32_t)t2, (uint32_t)t1, p0, e20 + (n << 20), sign);
}
// a b, both normal, or (ZERO) a zero: the result is then +0
template <bool ZERO>
FST_HD double mul_int(double a, double b) {
  const W2 x = words(a), y = words(b);
  const uint32_t xh = mant_hi(x.h), yh = mant_hi(y.h);
  const uint64_t ll = (uint64_t)x.l * y.l;
  const uint64_t m1 = (uint64_t)xh * y.l + (ll >> 32);
  const uint64_t m2 = (uint64_t)x.l * yh + (uint32_t)m1;
  const uint64_t H = (uint64_t)xh * yh + (m1 >> 32) + (m2 >> 32);
  const uint32_t ex = x.h & 0x7FF00000u;
  const uint64_t r = round_product(H, (uint32_t)m2, (uint32_t)ll,
                                   ex + (y.h & 0x7FF00000u) - (1024u << 20),
                                   (x.h ^ y.h) & 0x80000000u);
  return of_bits(ZERO && ex == 0 ? 0 : r);
}
// a a, a normal or (ZERO) zero
template <bool ZERO>
FST_HD double sq_int(double a) {
  const W2 x = words(a);
  const uint32_t xh = mant_hi(x.h);
  const uint64_t ll = (uint64_t)x.l * x.l;
  const uint64_t m = (uint64_t)(2 * xh) * x.l + (ll >> 32);
  const uint64_t H = (uint64_t)xh * xh + (m >> 32);
  const uint32_t ex = x.h & 0x7FF00000u;
  const uint64_t r = round_product(H, (uint32_t)m, (uint32_t)ll, 2 * ex - (1024u << 20), 0);
  return of_bits(ZERO && ex == 0 ? 0 : r);
}
// mantissa and exponent of a positive constant
struct CK {
  uint64_t m;  // 53 bits
  int e;       // unbiased
};
#if defined(__CUDACC__)
__host__ __device__
#endif
constexpr CK const_of(double c) {
  int e = 0;
  while (c >= 2.0) { c *= 0.5; ++e; }
  while (c < 1.0) { c *= 2.0; --e; }
  return {(uint64_t)(c * 4503599627370496.0), e};
}
// c a for a constant c > 0, a normal or zero (the result is then +0).  A
// constant of at most 32 significant bits takes two multiplications.
template <class C>
FST_HD double mul_const(double a) {
  constexpr CK k = const_of(C::value);
  const W2 x = words(a);
  const uint32_t xh = mant_hi(x.h), ex = x.h & 0x7FF00000u, sg = x.h & 0x80000000u;
  const uint32_t e20 = ex + ((uint32_t)(k.e - 1) << 20);
  uint64_t r;
  if constexpr ((k.m & 0x1FFFFFull) == 0) {
    constexpr uint32_t y = (uint32_t)(k.m >> 21);  // [2^31, 2^32)
    const uint64_t t = (uint64_t)x.l * y;
    const uint64_t H = (uint64_t)xh * y + (t >> 32);  // 85 bits: (H, t's low word), [2^83, 2^85)
    const uint32_t n = (uint32_t)(H >> 52);
    // M = P >> (31 + n), its fraction to 32 bits: no lower bits remain
    const uint32_t q = 2u >> n;
    const uint64_t t0 = (uint64_t)(uint32_t)t * q;
    const uint64_t t1 = (uint64_t)(uint32_t)H * q + (t0 >> 32);
    const uint32_t m1 = (uint32_t)(H >> 32) * q + (uint32_t)(t1 >> 32);
    r = round_join(m1, (uint32_t)t1, (uint32_t)t0, 0, e20 + (n << 20), sg);
  } else {
    constexpr uint32_t yh = (uint32_t)(k.m >> 32), yl = (uint32_t)k.m;
    const uint64_t ll = (uint64_t)x.l * yl;
    const uint64_t m1 = (uint64_t)xh * yl + (ll >> 32);
    const uint64_t m2 = (uint64_t)x.l * yh + (uint32_t)m1;
    const uint64_t H = (uint64_t)xh * yh + (m1 >> 32) + (m2 >> 32);
    r = round_product(H, (uint32_t)m2, (uint32_t)ll, e20, sg);
  }
  return of_bits(ex == 0 ? 0 : r);
}
// the quotient's mantissa rounded (no ties, see div_by), joined to the exponent
// field e20 of a quotient below 1
FST_HD uint64_t round_quot(uint64_t q, uint32_t e20, uint32_t sign) {
  const uint32_t t = (uint32_t)(q >> 55);  // 1: 56 bits
  const uint32_t k = 0x40000000u >> t;     // M = q >> (2 + t)
  const uint64_t t0 = (uint64_t)(uint32_t)q * k;
  const uint64_t m = (uint64_t)(uint32_t)(q >> 32) * k + (t0 >> 32);
  const uint64_t r = (m + ((uint64_t)(e20 + (t << 20)) << 32)) + ((uint32_t)t0 >> 31);
  return r | ((uint64_t)sign << 32);
}
// c / b for a constant c > 0 and b > 0 normal, the quotient normal
template <class C>
FST_HD double div_const(double b) {
  constexpr CK k = const_of(C::value);
  const W2 y = words(b);
  const uint32_t bh = mant_hi(y.h);
  const uint64_t q =
      quot55((uint32_t)(k.m >> 32), (uint32_t)k.m, bh, y.l, recip32(bh, y.l));
  return of_bits(round_quot(q, ((2044u + (uint32_t)k.e) << 20) - (y.h & 0x7FF00000u), 0));
}


// a b rounded as IEEE for every input: the integer product where both are normal
// (or one is zero and the other normal or zero) and the result is normal, the
// operator elsewhere.
FST_HD double mul_rn(double a, double b) {
  const W2 x = words(a), y = words(b);
  const uint32_t ex = (x.h >> 20) & 0x7FFu, ey = (y.h >> 20) & 0x7FFu;
  const bool zx = ((x.h << 1) | x.l) == 0, zy = ((y.h << 1) | y.l) == 0, zero = zx || zy;
  const uint32_t sg = (x.h ^ y.h) & 0x80000000u;
  if ((!zx && ex - 1u >= 2046u) || (!zy && ey - 1u >= 2046u) ||
      (!zero && ex + ey - 1025u >= 2044u))
    return mul_any(a, b);
  const uint32_t xh = mant_hi(x.h), yh = mant_hi(y.h);
  const uint64_t ll = (uint64_t)x.l * y.l;
  const uint64_t m1 = (uint64_t)xh * y.l + (ll >> 32);
  const uint64_t m2 = (uint64_t)x.l * yh + (uint32_t)m1;
  const uint64_t H = (uint64_t)xh * yh + (m1 >> 32) + (m2 >> 32);
  const uint64_t r = round_product(H, (uint32_t)m2, (uint32_t)ll, (ex + ey - 1024u) << 20, sg);
  return of_bits(zero ? (uint64_t)sg << 32 : r);
}

#if defined(__CUDACC__)
// mul_rn, div_by and a/d as calls, for long straight-line kernels: inlined, a
// few dozen of them overflow the instruction caches, and the warps wait for
// instructions more than for anything else.
__device__ __noinline__ static double mul_call(double a, double b) { return mul_rn(a, b); }
__device__ __noinline__ static double div_call(double a, uint32_t hi, uint32_t lo, uint32_t R) {
  return div_by(a, Recip{hi, lo, R});
}
// three quotients in one call, side by side (div_exact)
struct Quot3 {
  double x, y, z;
};
__device__ __noinline__ static Quot3 div3_call(double a, double b, double c, Recip ra, Recip rb, Recip rc) {
  const Quot3 q{div_core(a, ra), div_core(b, rb), div_core(c, rc)};
  if (div_exact(a, ra) & div_exact(b, rb) & div_exact(c, rc)) return q;
  return {div_by(a, ra), div_by(b, rb), div_by(c, rc)};
}
#endif

}  // namespace fst64
