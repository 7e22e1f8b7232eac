// The elementary functions of csrc/spc_math.h against the C library's long
// double ones.  Prints the largest errors and "ok" when they are within the
// bounds that the roundings of the formulas give:
//  * sin, cos: the last sum rounds to half an ulp; before it five roundings of
//    numbers below 2^-5 (the reduced angle twice, its sine, two products), at
//    2^-59 each, and the series' rest, below 2^-60;
//  * -2 ln u: T and R are exact or below 2^-7 with T != 0, so half an ulp for
//    the last sum, at most that again for the sum before it where T = 0, and a
//    tenth for the rest;
//  * sqrt: half an ulp and the correction's remainder.
#include <cmath>
#include <cstdio>
#include <random>

#include "spc_math.h"

typedef long double ld;

static double ulp(double v) {
  int e;
  std::frexp(v, &e);
  return std::ldexp(1.0, e - 53);
}

int main() {
  std::mt19937_64 g(7);
  const ld two_pi = 6.283185307179586476925286766559005768L;
  double es = 0, ec = 0, et = 0, el = 0, eq = 0, en = 0;
  // what is left of a sine's or cosine's error after half an ulp, in 2^-58
  auto rest = [](ld want, double got) {
    return std::fmax(0.0, (double)(fabsl(want - got) - 0.5L * ulp((double)want)) * 0x1p58);
  };
  long long bad = 0;
  auto phase = [&](double x) {
    double s, c;
    spc::sincos_in_range(x, s, c);
    const ld S = sinl((ld)x), C = cosl((ld)x);
    es = std::fmax(es, rest(S, s));
    ec = std::fmax(ec, rest(C, c));
  };
  std::uniform_real_distribution<double> u(-1, 1);
  for (int k = 0; k < 1500000; ++k) {
    phase(3.2 * u(g));
    phase(1000.0 * u(g));
  }
  for (int k = -300; k <= 300; ++k)  // the table's points and the seams between them
    for (double d : {0.0, 1e-17, -1e-17, 1e-9, -1e-9, 1e-3, -1e-3}) phase((double)(two_pi * k / 256.0L) + d);
  double ew = 0;  // the whole range: absolute error against 2^-53
  for (int k = 0; k < 500000; ++k) {
    const double x = 1048575.0 * u(g);
    double s, c;
    spc::sincos_in_range(x, s, c);
    ew = std::fmax(ew, (double)std::fmax(fabsl(sinl((ld)x) - s), fabsl(cosl((ld)x) - c)));
  }
  auto draw = [&](std::uint64_t A, std::uint64_t b) {
    const double l = spc::neg2_log53(A), r = spc::sqrt_pos(l);
    // -2 ln(A 2^-53): by log1p near one, where 1 - A 2^-53 is exact
    const ld L = A > (1ull << 52) ? -2.0L * log1pl(-(ld)((1ull << 53) - A) * 0x1.0p-53L)
                                  : -2.0L * (logl((ld)A) - 53.0L * 0.693147180559945309417232121458176568L);
    if (A == 1ull << 53) {
      if (l != 0.0 || r != 0.0) ++bad;
    } else {
      el = std::fmax(el, (double)(fabsl(L - l) / ulp((double)L)));
      eq = std::fmax(eq, (double)(fabsl(sqrtl((ld)l) - r) / ulp(r)));
    }
    double s, c;
    spc::sincos_turn53(b, s, c);
    // the angle from the nearest quarter turn, exact in integers
    const std::uint64_t q = (b + (1ull << 50)) >> 51;
    const ld a = two_pi * (ld)(std::int64_t)(b - (q << 51)) * 0x1.0p-53L;
    const ld ca = cosl(a), sa = sinl(a);
    const ld C = q % 4 == 0 ? ca : q % 4 == 1 ? -sa : q % 4 == 2 ? -ca : sa;
    const ld S = q % 4 == 0 ? sa : q % 4 == 1 ? ca : q % 4 == 2 ? -sa : -ca;
    et = std::fmax(et, std::fmax(rest(S, s), rest(C, c)));
    const ld R = sqrtl(L);
    en = std::fmax(en, (double)std::fmax(fabsl(R * C - r * c), fabsl(R * S - r * s)) / ulp((double)R));
  };
  const std::uint64_t top = 1ull << 53;
  for (int k = 0; k < 1500000; ++k) {
    draw((g() >> 11) + 1, g() >> 11);
    draw((g() >> (11 + g() % 53)) + 1, g() >> 11);
    draw(top - (g() >> (11 + g() % 53)), (g() >> (11 + g() % 53)) & (top - 1));
  }
  for (std::uint64_t j = 0; j <= 256; ++j)  // the tables' points and seams
    for (int d = -1; d <= 1; ++d) {
      const std::uint64_t b = ((j << 45) + (std::uint64_t)d) & (top - 1);
      draw(b ? b : 1, b);
      draw(top - (b >> 1), b);
    }
  for (int k = 0; k < 3000000; ++k) {
    const int q = 11 + (int)(g() % 42);
    const double v = std::ldexp(u(g), 51 - q - (int)(g() % 60));
    const double h = std::ldexp((double)((long long)(g() % 2001) - 1000) + 0.5, -q);  // ties
    for (double x : {v, h})
      if (spc::double_to_fixed(x, q) != std::llrint(std::ldexp(x, q))) ++bad;
  }
  for (double x : {0.0, -0.0, 1.0, -1.0, 5e-324})
    if (spc::double_to_fixed(x, 51) != std::llrint(std::ldexp(x, 51))) ++bad;
  std::printf("sin %.3f cos %.3f turn %.3f 2^-58; log %.3f sqrt %.3f ulp; normals %.3f ulp of the radius; "
              "|x| < 2^20 %.3g; %lld integers differ\n", es, ec, et, el, eq, en, ew, bad);
  const bool ok = es <= 2.7 && ec <= 2.7 && et <= 2.7 && el <= 1.1 && eq <= 0.51 && en <= 2.5 && ew <= 1.2e-16 && !bad;
  std::printf(ok ? "ok\n" : "FAILED\n");
  return ok ? 0 : 1;
}
