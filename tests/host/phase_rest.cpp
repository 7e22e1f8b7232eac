// sincos_with_rest (csrc/spc_math.h): the sine and cosine are sincos_in_range's, and
// the rest is the angle between the phase and the rounded pair.  What is left of
// its error: the cosine's series (d^8 / 40320 for |d| <= pi / 128, turned by d:
// 2^-63.4) and two roundings of numbers below 2^-11 (2^-64 each); with the four
// products here (2^-65 each where long double has 64 bits) below 2^-61.8.
#include <cmath>
#include <cstdio>
#include <random>

#include "spc_math.h"

typedef long double ld;

constexpr double kBound = 0x1.26p-62;

int main() {
  std::mt19937_64 g(5);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  double worst = 0.0, largest = 0.0;
  long long differ = 0;
  auto check = [&](double ph) {
    double s, c, s0, c0, rest;
    int k;
    spc::sincos_in_range(ph, s0, c0);
    spc::sincos_with_rest(ph, s, c, k, rest);
    if (s != s0 || c != c0) ++differ;
    const double n = std::rint(ph * 20.371832715762602);
    if (((int)n & 127) != k) return;  // between two points: either will do
    // the reduced phase: its first part is exact in double
    const ld d = (ld)std::fma(-n, 0x1.921fb54442d18p-5, ph) - (ld)n * 0x1.1a62633145c07p-59L;
    // the pair turned back by the table's point (its angle is exact there) lies at
    // atan2(sine, cosine) = d - rest
    const spc::double4_t p = spc::kCircle[k];
    const ld sn = ((ld)s * p.x - (ld)c * p.y) + ((ld)s * p.z - (ld)c * p.w);
    const ld cs = ((ld)c * p.x + (ld)s * p.y) + ((ld)c * p.z + (ld)s * p.w);
    const ld want = d - atan2l(sn, cs);
    largest = std::fmax(largest, std::fabs(rest));
    worst = std::fmax(worst, (double)fabsl(want - rest));
  };
  for (int k = 0; k < 400000; ++k) {
    check(3.2 * u(g));
    check(300.0 * u(g));
    check(std::ldexp(u(g), (int)(g() % 60) - 45));
  }
  std::printf("rest up to 2^%.2f, error 2^%.2f; %lld values differ\n", std::log2(largest), std::log2(worst), differ);
  const bool ok = worst <= kBound && largest <= 0x1.9p-54 && differ == 0;
  std::printf(ok ? "ok\n" : "FAILED\n");
  return ok ? 0 : 1;
}
