// Elementary functions of the per-particle work, by few double operations.
//
// GB300 runs double arithmetic at 1/64 of the FP32 rate (one warp instruction
// takes 16 cycles of an SM), so a particle's sines, cosines and normals cost
// more than all of its neighbour tests where cells are sparse: the 96-system
// FP32X ensemble spent 62% of its neighbour pass and most of its gather on the
// FP64 pipe.  What integer instructions can do (scaling by powers of two,
// splitting off exponents, rounding to fixed point) is done with them here,
// and the functions are table-driven with short Taylor polynomials:
//  * sin and cos: reduction to the nearest of 128 points of the circle, kept
//    to twice double precision, and the angle-addition formulas; 18 double
//    operations for both.  P. T. P. Tang, "Table-lookup algorithms for
//    elementary functions and their error analysis", ARITH-10, 1991;
//  * -2 ln u for u = A 2^-53: the nearest of 129 points of [1, 2], ln(1 + r)
//    by its series; 13 operations.  P. T. P. Tang, "Table-driven
//    implementation of the logarithm function in IEEE floating-point
//    arithmetic", ACM TOMS 16(4), 1990;
//  * the square root: the hardware's reciprocal square root estimate, one
//    Goldschmidt step and a correction by the exact remainder (P. Markstein,
//    IBM J. Res. Dev. 34(1), 1990); 6 operations.
// Errors (tests/test_math_accuracy.py on the CPU, tests/test_gpu_math_device.py
// on the GPU): sin and cos within half an ulp plus 2.7 2^-58 (the sum of the
// roundings on the way, all below 2^-5), -2 ln u within 1.1 ulp (largest found
// 0.998, mean 0.250, that of a correctly rounded one; CUDA's log: 1 ulp), the
// square root within 0.51 (0.5000 on the GPU).
// Before and after, FP32X step of that ensemble: 353 -> 293 us.
// Plain C++ as well, for those tests.
#pragma once

#include <cmath>
#include <cstdint>

#include "spc_fixed.h"

#if defined(__CUDACC__)
#define SPC_MATH_FN __device__ __forceinline__
#define SPC_TABLE(T, name, n) static __device__ const T name[n]
#else
#define SPC_MATH_FN inline
#define SPC_TABLE(T, name, n) static const T name[n]
#endif

namespace spc {

struct alignas(32) double4_t {
  double x, y, z, w;
};

}  // namespace spc

#include "spc_tables.h"

namespace spc {

SPC_MATH_FN double fma_rn(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
  return __fma_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}
SPC_MATH_FN double mul_rn(double a, double b) {
#if defined(__CUDA_ARCH__)
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}
SPC_MATH_FN double add_rn(double a, double b) {
#if defined(__CUDA_ARCH__)
  return __dadd_rn(a, b);
#else
  return a + b;
#endif
}
SPC_MATH_FN std::uint64_t double_to_bits(double d) {
#if defined(__CUDA_ARCH__)
  return static_cast<std::uint64_t>(__double_as_longlong(d));
#else
  std::uint64_t b;
  __builtin_memcpy(&b, &d, sizeof b);
  return b;
#endif
}

constexpr double kRoundMagic = 6755399441055744.0;  // 1.5 2^52: the sum's low bits are the rounded integer

// cos and sin of 2 pi k / 128 + d, |d| <= pi / 128.
SPC_MATH_FN void circle_point(int k, double d, double &s, double &c) {
  const double4_t p = kCircle[k & 127];
  const double d2 = mul_rn(d, d);
  // cos d - 1 and sin d (terms up to d^6 / 720 and d^7 / 5040)
  const double cm1 = mul_rn(d2, fma_rn(d2, fma_rn(d2, -1.0 / 720.0, 1.0 / 24.0), -0.5));
  const double sn = fma_rn(mul_rn(d, d2), fma_rn(d2, fma_rn(d2, -1.0 / 5040.0, 1.0 / 120.0), -1.0 / 6.0), d);
  c = add_rn(p.x, fma_rn(p.x, cm1, fma_rn(-p.y, sn, p.z)));
  s = add_rn(p.y, fma_rn(p.y, cm1, fma_rn(p.x, sn, p.w)));
}

// sin and cos of a phase.  The reduction by 2 pi / 128 in two parts is exact
// enough below 2^20; larger (or not finite) phases go to the library function.
SPC_MATH_FN bool phase_in_range(double ph) {
  return (static_cast<std::uint32_t>(double_to_bits(ph) >> 32) & 0x7fffffffu) < 0x41300000u;
}
SPC_MATH_FN void sincos_in_range(double ph, double &s, double &c) {
  const double t = fma_rn(ph, 0x1.45f306dc9c883p+4, kRoundMagic);  // 64 / pi
  const double n = add_rn(t, -kRoundMagic);
  double d = fma_rn(-n, 0x1.921fb54442d18p-5, ph);
  d = fma_rn(-n, 0x1.1a62633145c07p-59, d);
  circle_point(static_cast<int>(double_to_bits(t)), d, s, c);
}

// The same sine and cosine, bit for bit, with the point's number k and the angle
// `rest` by which the phase exceeds that of the rounded pair (|rest| < 2^-53.4,
// within 2^-62): every rounding on the way kept as a second double.  28 more
// operations.
SPC_MATH_FN void sincos_with_rest(double ph, double &s, double &c, int &k, double &rest) {
  const double t = fma_rn(ph, 0x1.45f306dc9c883p+4, kRoundMagic);  // 64 / pi
  const double n = add_rn(t, -kRoundMagic);
  const double d1 = fma_rn(-n, 0x1.921fb54442d18p-5, ph);  // exact
  const double d = fma_rn(-n, 0x1.1a62633145c07p-59, d1);
  const double dl = fma_rn(-n, 0x1.1a62633145c07p-59, add_rn(d1, -d));
  k = static_cast<int>(double_to_bits(t)) & 127;
  const double4_t p = kCircle[k];
  const double d2 = mul_rn(d, d), d3 = mul_rn(d, d2);
  const double cm1 = mul_rn(d2, fma_rn(d2, fma_rn(d2, -1.0 / 720.0, 1.0 / 24.0), -0.5));
  const double q = fma_rn(d2, fma_rn(d2, -1.0 / 5040.0, 1.0 / 120.0), -1.0 / 6.0);
  const double sn = fma_rn(d3, q, d);
  const double snl = add_rn(fma_rn(d3, q, add_rn(d, -sn)), dl);
  const double ic = fma_rn(-p.y, sn, p.z), is = fma_rn(p.x, sn, p.w);
  const double wc = fma_rn(p.x, cm1, ic), ws = fma_rn(p.y, cm1, is);
  c = add_rn(p.x, wc);
  s = add_rn(p.y, ws);
  const double icl = fma_rn(-p.w, sn, add_rn(fma_rn(-p.y, sn, -ic), p.z));
  const double isl = fma_rn(p.z, sn, add_rn(fma_rn(p.x, sn, -is), p.w));
  const double wcl = add_rn(fma_rn(p.x, cm1, add_rn(ic, -wc)), fma_rn(-p.y, snl, icl));
  const double wsl = add_rn(fma_rn(p.y, cm1, add_rn(is, -ws)), fma_rn(p.x, snl, isl));
  const double cl = add_rn(add_rn(add_rn(p.x, -c), wc), wcl), sl = add_rn(add_rn(add_rn(p.y, -s), ws), wsl);
  rest = fma_rn(c, sl, -mul_rn(s, cl));
}

// RN(v 2^q) for |v 2^q| < 2^31, by one addition.
SPC_MATH_FN int small_to_int(double v, int q) {
  return static_cast<int>(double_to_bits(add_rn(v, kRoundMagic * pow2i(-q))));
}

// cos and sin of 2 pi b 2^-53, b < 2^53.
SPC_MATH_FN void sincos_turn53(std::uint64_t b, double &s, double &c) {
  const std::uint64_t k = (b + (1ull << 45)) >> 46;
  const std::int64_t rest = static_cast<std::int64_t>(b - (k << 46));  // |rest| <= 2^45
  const double r = add_rn(bits_to_double(0x4338000000000000ull + static_cast<std::uint64_t>(rest)), -kRoundMagic);
  circle_point(static_cast<int>(k), mul_rn(r, 0x1.921fb54442d18p-51), s, c);  // 2 pi 2^-53
}

// -2 ln(A 2^-53), 1 <= A <= 2^53.
SPC_MATH_FN double neg2_log53(std::uint64_t A) {
  const int e = 63 - clz_u64(A);                                   // A = 2^e m
  const std::uint64_t f = (A << (63 - e)) << 1 >> 12;              // m's fraction bits
  const double m = bits_to_double(0x3ff0000000000000ull | f);
  const int i = static_cast<int>((f + (1ull << 44)) >> 45);        // nearest of 128 steps of [1, 2]
  const double4_t p = kLog[i];
  const int K = 53 - e - (i > 64 ? 1 : 0);
  const double Kd = add_rn(bits_to_double(0x4330000000000000ull + static_cast<std::uint64_t>(K)), -4503599627370496.0);
  const double R = fma_rn(m, p.x, 2.0);                            // -2 r, m = C' (1 + r)
  const double R2 = mul_rn(R, R);
  // -2 ln(1 + r) = R + R^2 / 4 + R^3 / 12 + R^4 / 32 + R^5 / 80 + R^6 / 192 + R^7 / 448
  double q = fma_rn(R, 1.0 / 448.0, 1.0 / 192.0);
  q = fma_rn(R, q, 1.0 / 80.0);
  q = fma_rn(R, q, 1.0 / 32.0);
  q = fma_rn(R, q, 1.0 / 12.0);
  q = fma_rn(R, q, 0.25);
  // 2 ln 2 per power of two, a multiple of 2^-44 and the rest: T is exact
  const double T = fma_rn(Kd, 0x1.62e42fefa3ap+0, p.y);
  const double low = fma_rn(R2, q, fma_rn(Kd, -0x1.0ca86c3898dp-48, p.z));
  return add_rn(T, add_rn(R, low));
}

// sqrt(x), x = 0 or 2^-900 < x < 2^1000 (the remainder of the last step is then
// normal).
SPC_MATH_FN double sqrt_pos(double x) {
#if defined(__CUDA_ARCH__)
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
#else
  const double y = 1.0f / std::sqrt(static_cast<float>(x));
#endif
  double g = mul_rn(x, y);
  double h = bits_to_double(double_to_bits(y) - (1ull << 52));  // y / 2
  const double r = fma_rn(-g, h, 0.5);
  g = fma_rn(g, r, g);
  h = fma_rn(h, r, h);
  g = fma_rn(fma_rn(-g, g, x), h, g);
  return x == 0.0 ? 0.0 : g;
}

// RN(v 2^q) as an integer: to nearest, ties to even, by integer instructions
// (the scaling is exact, so this is the rounding of the scaled value).
// kNotFixed when v is not finite or |v 2^q| is 2^62 or more.
constexpr long long kNotFixed = -0x7fffffffffffffffll - 1;
SPC_MATH_FN long long double_to_fixed(double v, int q) {
  const std::uint64_t b = double_to_bits(v);
  const int e = static_cast<int>((b >> 52) & 0x7ff);
  const int drop = 1075 - e - q;  // bits below the unit
  if (e == 0x7ff || drop < -9) return kNotFixed;
  if (drop > 54 || e == 0) return 0;
  const std::uint64_t m = (b & 0xfffffffffffffull) | (1ull << 52);
  std::uint64_t r = drop < 0 ? m << -drop : m;
  if (drop > 0) {
    r = m >> drop;
    const std::uint64_t rest = m << (64 - drop), half = 1ull << 63;
    r += (rest > half || (rest == half && (r & 1ull))) ? 1ull : 0ull;
  }
  return (b >> 63) ? -static_cast<long long>(r) : static_cast<long long>(r);
}

}  // namespace spc
