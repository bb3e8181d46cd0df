// IEEE FP64 multiplication, division, reciprocal, square root and the
// conversion to FP32, round to nearest even, in integer arithmetic.
//
// Why: GB300's FP64 pipe takes a warp instruction every ~80 cycles per SM
// sub-partition, however many lanes are active, while the integer and FP32
// pipes issue one per cycle or two.  A product below is about 35 integer
// instructions, a quotient or root 50 to 90 against 8 to 20 FP64 ones, so the
// ray state's arithmetic runs several times faster when the products go here
// and only the additions stay on the FP64 pipe, and the two overlap.  The
// results are the correctly rounded ones, i.e. the same bits.
//
// Range: operands are zero or normal with exponents the caller has checked
// (safe64), far enough from the limits that no result is subnormal or
// overflows; everything else takes the hardware's instructions.  The methods
// are the textbook ones: a 53 x 53 bit integer product rounded once; a
// Newton iteration in 64-bit fixed point from an FP32 seed, whose candidate
// is settled by its exact remainder (Markstein 1990; Knuth, TAOCP 4.3.1).
//
// Host code compiles it too (the tests compare it with the host's own FP64).
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define SBR_HD __host__ __device__ __forceinline__
#else
#define SBR_HD inline
#endif

namespace sbr {
namespace soft64 {

SBR_HD uint64_t bits(double x) {
#ifdef __CUDA_ARCH__
  return uint64_t(__double_as_longlong(x));
#else
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return u;
#endif
}
SBR_HD double from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  std::memcpy(&x, &u, 8);
  return x;
#endif
}
SBR_HD float f32_bits(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  std::memcpy(&x, &u, 4);
  return x;
#endif
}
SBR_HD uint64_t mulhi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return uint64_t((unsigned __int128)a * b >> 64);
#endif
}
// FP32 seeds, within 2^-22 of 1/x and 1/sqrt(x) for x in [1, 4).
#ifndef SBR_SOFT64_SEED_ERROR  // the tests widen the host's seeds
#define SBR_SOFT64_SEED_ERROR 0.0f
#endif
SBR_HD float seed_rcp(float x) {
#ifdef __CUDA_ARCH__
  return __fdividef(1.0f, x);
#else
  return (1.0f / x) * (1.0f + SBR_SOFT64_SEED_ERROR);
#endif
}
SBR_HD float seed_rsqrt(float x) {
#ifdef __CUDA_ARCH__
  return rsqrtf(x);
#else
  return float(1.0 / __builtin_sqrt(double(x))) * (1.0f + SBR_SOFT64_SEED_ERROR);
#endif
}

// Zero, or a magnitude in [2^-120, 2^100): sums and products of a few such
// values (the triangle test, a reflection, a normalisation) stay zero or
// normal, also after cancellation.
SBR_HD bool safe(double x) {
  const uint64_t u = bits(x);
  const uint32_t e = uint32_t(u >> 32) & 0x7fffffffu;
  return e - (uint32_t(1023 - 120) << 20) < (220u << 20) || (u << 1) == 0;
}

// x < 0, x > c (c > 0) and |x| < c as the FP64 comparisons decide them (NaN:
// false), by integer comparison: an FP64 comparison takes an FP64 pipe slot.
constexpr uint64_t kInf = 0x7ff0000000000000ull;
SBR_HD bool negative(double x) {
  const uint64_t u = bits(x), m = u & ~(1ull << 63);
  return (u >> 63) && m != 0 && m <= kInf;
}
SBR_HD bool above(double x, double c) {
  const uint64_t u = bits(x);
  return u - bits(c) - 1 < kInf - bits(c);  // bits(c) < u <= inf
}
SBR_HD bool magnitude_below(double x, double c) {
  return (bits(x) & ~(1ull << 63)) < bits(c);
}
// a < b and a == b for a, b >= +0 or NaN (a NaN on the left: false).
SBR_HD bool less(double a, double b) { return bits(a) < bits(b); }
SBR_HD bool same(double a, double b) { return bits(a) == bits(b); }

SBR_HD double mul(double a, double b) {
  const uint64_t ua = bits(a), ub = bits(b);
  const uint32_t ah = uint32_t(ua >> 32), bh = uint32_t(ub >> 32);
  // a's 53 bits at the top of 64, b's shifted up by one: bits 64.. of the
  // product are the result's mantissa with 0 (c = 0) or 1 (c = 1) bit more
  const uint64_t A = (ua << 11) | (1ull << 63);
  const uint64_t B = ((ub << 1) & 0x001fffffffffffffull) | (1ull << 53);
  const uint32_t a0 = uint32_t(A), a1 = uint32_t(A >> 32);
  const uint32_t b0 = uint32_t(B), b1 = uint32_t(B >> 32);
  const uint64_t p = uint64_t(a0) * b0;
  const uint64_t t = uint64_t(a1) * b0 + (p >> 32);
  const uint64_t u = uint64_t(a0) * b1 + uint32_t(t);
  uint64_t h = uint64_t(a1) * b1 + (t >> 32) + (u >> 32);
  const uint32_t l0 = uint32_t(p), l1 = uint32_t(u);
  const uint32_t c = uint32_t(h >> 53);
  // the bits below the mantissa: the first one (sign of r1) and the rest
#ifdef __CUDA_ARCH__
  const uint32_t r1 = __funnelshift_r(l1, uint32_t(h), c);
#else
  const uint32_t r1 = c ? (l1 >> 1 | uint32_t(h) << 31) : l1;
#endif
  h >>= c;
  const uint32_t rest = (r1 & 0x7fffffffu) | l0 | (l1 & c) | (uint32_t(h) & 1u);
  h += (int32_t(r1) < 0 && rest != 0) ? 1 : 0;
  const uint32_t ea = ah & 0x7ff00000u, eb = bh & 0x7ff00000u;
  const uint32_t hi = uint32_t(h >> 32) + ea + eb - (1024u << 20) + (c << 20);
  const uint32_t sg = (ah ^ bh) & 0x80000000u;
  const bool z = ea == 0 || eb == 0;
  return from_bits(uint64_t(z ? sg : (hi | sg)) << 32 | (z ? 0u : uint32_t(h)));
}

// 1/m in Q63 for the mantissa m in [1, 2), M = m 2^63: within 2^-60.
SBR_HD uint64_t rcp_q63(uint64_t M) {
  const uint32_t mh = uint32_t(M >> 32), ml = uint32_t(M);
  const float r = seed_rcp(f32_bits(0x3f800000u | ((mh >> 8) & 0x7fffffu)));
  const uint32_t x0 = uint32_t(r * 2147483648.0f);  // Q31
  const uint64_t t0 = uint64_t(mh) * x0 + (uint64_t(ml) * x0 >> 32);  // m x0, Q62
  const int64_t e0 = int64_t((1ull << 62) - t0);  // |e0| < 2^-21: half of the 32 bits' range
  const uint64_t x1 = (uint64_t(x0) << 32) + uint64_t((int64_t(x0) * int32_t(e0 >> 11)) >> 19);
  const int32_t e1 = int32_t((1ull << 62) - mulhi(M, x1));  // |e1| < 2^-41
  return x1 + uint64_t((int64_t(x1 >> 32) * e1) >> 30);
}

// The candidate q of N / D (N, D integers, q within one of the quotient)
// moved to the nearest integer; d = N - q D, exact in 64 bits.
SBR_HD uint64_t nearest(uint64_t q, int64_t d, uint64_t D) {
  if (2 * d > int64_t(D)) return q + 1;
  if (2 * d < -int64_t(D)) return q - 1;
  return q;
}

// 1 / a, a nonzero.
SBR_HD double rcp(double a) {
  const uint64_t ua = bits(a);
  const uint64_t M = (ua << 11) | (1ull << 63), m53 = M >> 11;
  const uint64_t x = rcp_q63(M);
  uint64_t q = (x + 512) >> 10;  // 2^53 / m
  q = nearest(q, int64_t(0 - q * m53), m53);  // 2^105 = 0 mod 2^64
  const uint64_t ea = (ua >> 52) & 0x7ff;
  return from_bits(((2044 - ea) << 52) + q | (ua & (1ull << 63)));
}

// a / b given x = rcp_q63 of b's mantissa.
SBR_HD double div_by(double a, double b, uint64_t x) {
  const uint64_t ua = bits(a), ub = bits(b);
  const uint64_t A = (ua << 11) | (1ull << 63), D = (ub & 0x000fffffffffffffull) | (1ull << 52);
  const uint64_t t = mulhi(A, x);  // quotient of the mantissas, Q62
  const uint32_t one = uint32_t(t >> 62);  // 1: the quotient is at least 1
  uint64_t q = (t + (256ull << one)) >> (9 + one);
  const uint64_t N = (A >> 11) << (53 - one);  // mod 2^64
  q = nearest(q, int64_t(N - q * D), D);
  const uint32_t ea = uint32_t(ua >> 52) & 0x7ff, eb = uint32_t(ub >> 52) & 0x7ff;
  const uint64_t sg = (ua ^ ub) & (1ull << 63);
  const uint64_t r = (uint64_t(ea - eb + 1021 + one) << 52) + q;
  return from_bits(ea == 0 ? sg : (r | sg));
}
SBR_HD uint64_t rcp_of(double b) { return rcp_q63((bits(b) << 11) | (1ull << 63)); }
SBR_HD double div(double a, double b) { return div_by(a, b, rcp_of(b)); }

// sqrt(z), z >= +0.
SBR_HD double sqrt(double z) {
  const uint64_t u = bits(z);
  const uint32_t e = uint32_t(u >> 52);
  const uint32_t odd = (e & 1) ^ 1;  // exponent e - 1023 odd: w = 2 m, else w = m
  const uint64_t m53 = (u & 0x000fffffffffffffull) | (1ull << 52);
  const uint64_t W = m53 << (10 + odd);  // w in [1, 4), Q62
  const uint32_t wh = uint32_t(m53 >> 21);  // 32 bits: m's leading bits
  const float f = f32_bits((0x3f800000u + (odd << 23)) | ((wh >> 8) & 0x7fffffu));
  const uint32_t x0 = uint32_t(seed_rsqrt(f) * 2147483648.0f);          // 1/sqrt(w), Q31
  const int64_t e0 = int64_t((1ull << 60) - mulhi(W, uint64_t(x0) * x0));  // 1 - w x0^2, Q60
  const uint64_t x1 = (uint64_t(x0) << 32) + uint64_t((int64_t(x0) * int32_t(e0 >> 10)) >> 19);
  const uint64_t s1 = mulhi(W, x1);  // Q61
  const int32_t r = int32_t((W >> 4) - mulhi(s1, s1));  // w - s1^2, Q58
  const uint64_t s2 = s1 + uint64_t((int64_t(x1 >> 32) * r) >> 29);
  uint64_t q = (s2 + 256) >> 9;  // sqrt(w) 2^52
  const int64_t d = int64_t(((m53 << odd) << 52) - q * q);
  if (d > int64_t(q)) ++q;
  else if (d <= -int64_t(q)) --q;
  return from_bits((u << 1) == 0 ? 0 : (uint64_t((e + 1021) >> 1) << 52) + q);
}

// float(x), round to nearest even; outside FP32's normal range (zero
// excepted) the hardware converts.
SBR_HD float to_f32(double x) {
  const uint64_t u = bits(x);
  const uint32_t h = uint32_t(u >> 32), l = uint32_t(u), sg = h & 0x80000000u;
  const uint32_t e = h & 0x7ff00000u;
  if (e - (897u << 20) <= (253u << 20)) {
    const uint32_t t = uint32_t(u >> 29);  // FP32 mantissa and the exponent's low bits
    uint32_t r = (t & 0x7fffffffu) ^ 0x40000000u;
    r += ((l << 3) + (t & 1u) > 0x80000000u) ? 1u : 0u;
    return f32_bits(r | sg);
  }
  if (e == 0) return f32_bits(sg);
  return float(x);
}

// double(x) and double(n) (n in [0, 2^31)), exact; subnormal, infinite and NaN
// floats are left to the hardware.
SBR_HD double from_f32(float x) {
#ifdef __CUDA_ARCH__
  const uint32_t u = __float_as_uint(x);
#else
  uint32_t u;
  std::memcpy(&u, &x, 4);
#endif
  const uint32_t e = (u >> 23) & 0xffu;
  if (e - 1u < 254u)
    return from_bits(uint64_t((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20))) << 32 |
                     uint64_t(u << 29));
  if ((u << 1) == 0) return from_bits(uint64_t(u) << 32);
  return double(x);
}
SBR_HD double from_int(int n) {
  if (n == 0) return 0.0;
#ifdef __CUDA_ARCH__
  const int lead = __clz(n);
#else
  const int lead = __builtin_clz(unsigned(n));
#endif
  const uint64_t m = uint64_t(n) << (lead + 21);  // leading bit at 52
  return from_bits((uint64_t(1023 + 30 - lead) << 52) + m);  // its carry makes the exponent
}

}  // namespace soft64
}  // namespace sbr
