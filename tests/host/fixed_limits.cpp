// double_to_fixed (csrc/spc_math.h) outside the range of its usual values:
// not finite, and up to and beyond 2^62 units.
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
  std::printf(bad ? "FAILED\n" : "ok\n");
  return bad ? 1 : 0;
}
