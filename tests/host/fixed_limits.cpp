// double_to_fixed (csrc/spc_math.h) outside the range of its usual values:
// not finite, and up to and beyond 2^62 units; and fixed_to_double
// (csrc/spc_fixed.h) with units far above one.
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include <limits>

#include "spc_math.h"

int main() {
  int bad = 0;
  auto expect = [&](double v, int q, long long want) {
    if (spc::double_to_fixed(v, q) != want) {
      std::printf("%g at %d: %lld, not %lld\n", v, q, spc::double_to_fixed(v, q), want);
      ++bad;
    }
  };
  const double inf = std::numeric_limits<double>::infinity(), nan = std::nan("");
  for (int q : {52, 11, 0, -300}) {
    for (double v : {nan, -nan, inf, -inf}) expect(v, q, spc::kNotFixed);
    for (int e = -60; e < 62; ++e)
      for (double m : {1.0, -1.0, 1.25, -1.9999999999999998}) {
        const double v = std::ldexp(m, e - q);
        expect(v, q, std::llrint(std::ldexp(v, q)));
      }
    for (int e : {62, 63, 64, 200})
      for (double m : {1.0, -1.0}) expect(std::ldexp(m, e - q), q, spc::kNotFixed);
  }
  for (int q : {52, 0, -1, -300, -849})
    for (long long v : {1ll, -1ll, 3ll, (1ll << 52) + 1, (1ll << 62) + 129, -(1ll << 62) - 257})
      if (spc::fixed_to_double(v, q) != std::ldexp((double)v, -q)) ++bad;
  std::printf(bad ? "FAILED\n" : "ok\n");
  return bad ? 1 : 0;
}
