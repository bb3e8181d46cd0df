// FP64 operations in integer arithmetic (csrc/sbr_soft64.cuh) against the
// host's own, bit for bit: random and patterned mantissas, products and
// quotients next to a rounding boundary, perfect squares and their neighbours,
// zeros of both signs, FP32 conversions at ties and at the ends of its range,
// comparisons with NaN and infinities.  SBR_SOFT64_SEED_ERROR shifts the FP32
// seeds by more than the device's may err.  Exit status 0: no difference.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "sbr_soft64.cuh"

using namespace sbr;

static std::mt19937_64 rng(1);
static long bad = 0;

static double patterned() {
  uint64_t m = rng() & 0xfffffffffffffull;
  switch (rng() % 8) {
    case 0: m = 0; break;
    case 1: m = 0xfffffffffffffull; break;
    case 2: m &= ~0ull << (rng() % 52); break;
    case 3: m |= (1ull << (rng() % 52)) - 1; break;
    case 4: m = 1ull << (rng() % 52); break;
    case 5: m = 0xfffffffffffffull & ~(1ull << (rng() % 52)); break;
    default: break;
  }
  const uint64_t e = 1023 - 119 + rng() % 218, s = rng() & (1ull << 63);
  return soft64::from_bits(rng() % 64 ? (s | e << 52 | m) : s);
}

static void same(const char* what, double got, double want) {
  if (soft64::bits(got) != soft64::bits(want) && bad++ < 10)
    std::printf("%s: %a, want %a\n", what, got, want);
}
static void same_f(double x) {
  const float got = soft64::to_f32(x), want = float(x);
  if (std::memcmp(&got, &want, 4) && x == x && bad++ < 10)
    std::printf("float(%a): %a, want %a\n", x, got, want);
}
static void same_tests(double x) {
  for (double c : {1.0, 1.1920928955078125e-07})
    if (soft64::above(x, c) != (x > c) || soft64::magnitude_below(x, c) != (std::fabs(x) < c))
      ++bad;
  if (soft64::negative(x) != (x < 0)) ++bad;
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
  for (long i = 0; i < n; ++i) {
    const double a = patterned(), b = patterned();
    if (!soft64::safe(a) || !soft64::safe(b)) ++bad;
    same("product", soft64::mul(a, b), a * b);
    same("root", soft64::sqrt(std::fabs(a)), std::sqrt(std::fabs(a)));
    const double one = 1.0 + std::ldexp(double(int64_t(rng()) >> 40), -52);
    same("root near 1", soft64::sqrt(one), std::sqrt(one));
    if (b != 0) {
      same("quotient", soft64::div(a, b), a / b);
      same("reciprocal", soft64::rcp(b), 1.0 / b);
      const double up = std::nextafter(a * b, rng() & 1 ? 1e300 : -1e300);
      if (a != 0) same("quotient next to a value", soft64::div(up, b), up / b);
      const double sq = std::nextafter(b * b, rng() & 1 ? 1e300 : 0);
      same("root next to a square", soft64::sqrt(sq), std::sqrt(sq));
    }
    same_f(a);
    // FP32 ties and their neighbours, also at the ends of its exponent range
    uint64_t u = rng() & ~0x1fffffffull;
    u |= rng() % 3 == 0 ? 0x10000000ull : (rng() & 1 ? 0x0fffffffull : 0x10000001ull);
    if (rng() % 16 == 0) u = (u & ~(0x7ffull << 52)) | uint64_t(rng() & 1 ? 1150 : 897) << 52;
    if ((u >> 52 & 0x7ff) != 0x7ff) same_f(soft64::from_bits(u));
    same_tests(soft64::from_bits(rng()));
    same_tests(a);
    const uint32_t f = uint32_t(rng());
    float x;
    std::memcpy(&x, &f, 4);
    if (x == x) same("double of a float", soft64::from_f32(x), double(x));
    const int k = int(rng() & 0x7fffffff) >> (rng() % 31);
    same("double of a count", soft64::from_int(k), double(k));
  }
  for (int k : {0, 1, 2, 3, 0x7fffffff, 0x7ffffffe, 0x40000000, 0x3fffffff})
    same("double of a count", soft64::from_int(k), double(k));
  for (float x : {0.0f, -0.0f, 1.0f, 1.17549435e-38f, 3.4028235e38f, 1e-45f, INFINITY})
    same("double of a float", soft64::from_f32(x), double(x));
  for (double x : {0.0, -0.0, double(INFINITY), double(-INFINITY), double(NAN), -double(NAN), 1.0,
                   -1.0, 5e-324, -5e-324, 1.7e308, 1.1920928955078125e-07}) {
    same_tests(x);
    same_f(x);
  }
  for (double x : {5e-324, 1e-200, 1e31, double(INFINITY), double(NAN)})
    if (soft64::safe(x)) ++bad;
  std::printf("%ld differences\n", bad);
  return bad != 0;
}
