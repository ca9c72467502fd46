// The integer-pipe FP64 operations (fiesta_gb300/csrc/fst_fp64.cuh) on the host,
// against the CPU's IEEE arithmetic.  The reciprocal seed is perturbed by up to
// two units in its last place, more than the GPU's instruction is off.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <random>

static thread_local int seed_ulp = 0;
static float perturbed_rcp(float f) {
  float r = 1.0f / f;
  uint32_t b;
  memcpy(&b, &r, 4);
  b += seed_ulp;
  if (f > 1.0f && b > 0x3F7FFFFFu) b = 0x3F7FFFFFu;  // 1/f < 1
  memcpy(&r, &b, 4);
  return r;
}
#define FST_RCP_SEED_HOST perturbed_rcp
#include "../../fiesta_gb300/csrc/fst_fp64.cuh"

using namespace fst64;

template <bool F32>
struct C {
#define CONST(name, n, d) \
  struct name { static constexpr double value = F32 ? (double)((float)(n) / (float)(d)) : (double)(n) / (d); };
  CONST(c1312, 13.0, 12.0) CONST(c13, 1.0, 3.0) CONST(c76, 7.0, 6.0) CONST(c116, 11.0, 6.0)
  CONST(c56, 5.0, 6.0) CONST(three, 3.0, 1.0) CONST(w1, 0.1, 1.0) CONST(w2, 0.6, 1.0) CONST(w3, 0.3, 1.0)
};

static bool same(double a, double b) { return a == b || (a != a && b != b); }

extern "C" long long fp64_check(long long n, uint64_t seed) {
  std::mt19937_64 r(seed);
  long long bad = 0;
  auto mant = [&]() -> uint64_t {  // random mantissas, runs of zeros and ones, the ends
    uint64_t m = r();
    switch (r() % 5) {
      case 0: m &= ~0ull << (r() % 53); break;
      case 1: m |= (1ull << (r() % 53)) - 1; break;
      case 2: m = (r() & 1) ? (r() & 0xFF) : ~(r() & 0xFFull); break;
    }
    return (m & 0xFFFFFFFFFFFFFull) | (r() & 1) << 63;
  };
  auto within = [&](int lo, int hi) { return of_bits(mant() | (uint64_t)(1023 + lo + (int)(r() % (hi - lo + 1))) << 52); };
  const double edge[] = {0.0, -0.0, 1.0, -1.0, INFINITY, -INFINITY, NAN, 4.9e-324, 2.2250738585072014e-308,
                         1.7976931348623157e308, 1e-300, 1e300, 3.0, 0.1};
  for (double a : edge)
    for (double b : edge) bad += !same(a / b, div_rn(a, b)) + !same(a * b, mul_rn(a, b));
  for (double a : edge)
    for (int k = -900; k <= 900; k += 7) bad += !same(a * std::ldexp(1.0, k), scale2(a, k, std::ldexp(1.0, k)));
  for (long long q = 0; q < n; ++q) {
    seed_ulp = (int)(r() % 5) - 2;
    double a = r() % 3 ? within(-30, 30) : of_bits(mant() | (r() % 2048) << 52);
    double b = r() % 3 ? within(-30, 30) : of_bits(mant() | (r() % 2048) << 52);
    if (r() % 4 == 0) {  // quotients next to representable and half-way values
      a = b * within(0, 1);
      a = of_bits(bits_of(a) + r() % 5 - 2);
    }
    bad += !same(a / b, div_rn(a, b));
    bad += !same(a / b, div_by(a, recip_of(b)));
    bad += !same(a * b, mul_rn(a, b));
    bad += !same(a * 0.5, half(a)) + !same(a * 2.0, twice(a)) + !same(a * 8.0, eight(a));
    const int k = (int)(r() % 2000) - 1000;
    bad += !same(a * std::ldexp(1.0, k), scale2(a, k, std::ldexp(1.0, k)));
    // the products' ranges: a normal or zero, the result normal
    double x = within(-200, 200), y = within(-200, 200);
    if (r() % 40 == 0) x = 0.0;
    bad += !same(x * y, mul_int<true>(x, y));
    bad += !same(x * x, sq_int<true>(x));
    if (x != 0) bad += !same(x * y, mul_int<false>(x, y)) + !same(x * x, sq_int<false>(x));
    auto consts = [&](auto c) {
      using D = decltype(c);
      bad += !same(D::c1312::value * x, mul_const<typename D::c1312>(x));
      bad += !same(D::c13::value * x, mul_const<typename D::c13>(x));
      bad += !same(D::c76::value * x, mul_const<typename D::c76>(x));
      bad += !same(D::c116::value * x, mul_const<typename D::c116>(x));
      bad += !same(D::c56::value * x, mul_const<typename D::c56>(x));
      bad += !same(D::three::value * x, mul_const<typename D::three>(x));
      const double p = std::fabs(y);
      bad += !same(D::w1::value / p, div_const<typename D::w1>(p));
      bad += !same(D::w2::value / p, div_const<typename D::w2>(p));
      bad += !same(D::w3::value / p, div_const<typename D::w3>(p));
    };
    consts(C<true>{});
    consts(C<false>{});
  }
  return bad;
}
