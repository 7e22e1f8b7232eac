// The functions of csrc/spc_math.h as the GPU runs them.  The root is seeded by
// the hardware's estimate, so its error is measured here; the others are the
// same operations as on the CPU and have to give the same bits (math_host.cpp).
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "spc_math.h"

typedef long double ld;

static double ulp(double v) {
  int e;
  std::frexp(v, &e);
  return std::ldexp(1.0, e - 53);
}

// u = A 2^-53 over all magnitudes, near one, and at the table's points and seams
static std::vector<std::uint64_t> log_arguments() {
  std::mt19937_64 g(11);
  const std::uint64_t top = 1ull << 53;
  std::vector<std::uint64_t> v;
  for (int k = 0; k < 400000; ++k) {
    v.push_back((g() >> 11) + 1);
    v.push_back((g() >> (11 + g() % 53)) + 1);
    v.push_back(top - (g() >> (11 + g() % 53)));
  }
  for (std::uint64_t j = 0; j <= 256; ++j)
    for (int s = 0; s < 8; ++s)
      for (int d = -1; d <= 1; ++d) {
        const std::uint64_t b = (((j + 256) << 44) >> s) + (std::uint64_t)d;
        if (b >= 1 && b <= top) v.push_back(b);
      }
  return v;
}
// squares of distances (1e-30 and less to L^2) and radii
static std::vector<double> root_arguments() {
  std::mt19937_64 g(12);
  std::uniform_real_distribution<double> m(1.0, 2.0);
  std::vector<double> v = {0.0};
  for (int k = 0; k < 600000; ++k) {
    v.push_back(std::ldexp(m(g), -(int)(g() % 120)));
    v.push_back(std::ldexp(m(g), (int)(g() % 1800) - 900));
    const double r = std::ldexp(m(g), (int)(g() % 40) - 20);
    v.push_back(r * r);
  }
  return v;
}

// -2 ln(A 2^-53): by log1p near one, else m 2^K with m in [sqrt(1/2), sqrt(2))
// and ln 2 as a short part, whose multiples are exact, and the rest
static ld neg2_log(std::uint64_t A) {
  const std::uint64_t top = 1ull << 53;
  if (A > top / 2) return -2.0L * log1pl(-(ld)(top - A) * 0x1.0p-53L);
  int K;
  ld m = frexpl((ld)A, &K);
  if (m < 0.70710678118654752440L) {
    m *= 2.0L;
    --K;
  }
  K -= 53;
  return -2.0L * (K * 0x1.62e42fep-1L + (logl(m) + K * 0x1.f473de6af278ece6p-30L));
}

// the worst error of l[k] = -2 ln(a[k] 2^-53), in ulp
static double log_error(const std::vector<std::uint64_t> &a, const std::vector<double> &l) {
  double worst = 0.0;
  for (std::size_t k = 0; k < a.size(); ++k) {
    const std::uint64_t A = a[k], top = 1ull << 53;
    if (A == top) {
      if (l[k] != 0.0) worst = HUGE_VAL;
      continue;
    }
    const ld L = neg2_log(A);
    worst = std::fmax(worst, (double)(fabsl(L - l[k]) / ulp((double)L)));
  }
  return worst;
}
static double root_error(const std::vector<double> &x, const std::vector<double> &r) {
  double worst = 0.0;
  for (std::size_t k = 0; k < x.size(); ++k) {
    if (x[k] == 0.0) {
      if (r[k] != 0.0) worst = HUGE_VAL;
      continue;
    }
    const ld R = sqrtl((ld)x[k]);
    worst = std::fmax(worst, (double)(fabsl(R - r[k]) / ulp((double)R)));
  }
  return worst;
}
constexpr double kLogBound = 1.1, kRootBound = 0.51;  // as on the CPU (math_accuracy.cpp)

double host_log(std::uint64_t A);
void host_sincos(double x, double &s, double &c);
void host_turn(std::uint64_t b, double &s, double &c);

__global__ void k_log(int n, const unsigned long long *a, double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = spc::neg2_log53(a[i]);
}
__global__ void k_root(int n, const double *x, double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = spc::sqrt_pos(x[i]);
}
__global__ void k_sincos(int n, const double *x, double *s, double *c) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) spc::sincos_in_range(x[i], s[i], c[i]);
}
__global__ void k_turn(int n, const unsigned long long *b, double *s, double *c) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) spc::sincos_turn53(b[i] >> 11, s[i], c[i]);
}

template <class T>
static T *managed(std::size_t n) {
  T *p = nullptr;
  if (cudaMallocManaged(&p, n * sizeof(T)) != cudaSuccess) {
    std::printf("no memory\n");
    std::exit(2);
  }
  return p;
}
template <class T>
static T *on_device(const std::vector<T> &v) {
  T *p = managed<T>(v.size());
  std::memcpy(p, v.data(), v.size() * sizeof(T));
  return p;
}
static std::vector<double> fetched(const double *p, std::size_t n) { return std::vector<double>(p, p + n); }
static bool same(double a, double b) { return std::memcmp(&a, &b, sizeof a) == 0; }

int main() {
  long long differ = 0;
  const auto blocks = [](std::size_t n) { return (int)((n + 255) / 256); };
  std::vector<unsigned long long> a;
  for (std::uint64_t A : log_arguments()) a.push_back(A);
  const std::vector<double> x = root_arguments();
  std::vector<double> ph;
  std::vector<unsigned long long> turns;
  std::mt19937_64 g(13);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  for (int k = 0; k < 500000; ++k) {
    ph.push_back(3.2 * u(g));
    ph.push_back(std::ldexp(u(g), (int)(g() % 60) - 40));
    turns.push_back(g());
  }
  double *l = managed<double>(a.size()), *r = managed<double>(x.size());
  double *s = managed<double>(ph.size()), *c = managed<double>(ph.size());
  double *ts = managed<double>(turns.size()), *tc = managed<double>(turns.size());
  k_log<<<blocks(a.size()), 256>>>((int)a.size(), on_device(a), l);
  k_root<<<blocks(x.size()), 256>>>((int)x.size(), on_device(x), r);
  k_sincos<<<blocks(ph.size()), 256>>>((int)ph.size(), on_device(ph), s, c);
  k_turn<<<blocks(turns.size()), 256>>>((int)turns.size(), on_device(turns), ts, tc);
  const cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    std::printf("%s\n", cudaGetErrorString(e));
    return 2;
  }
  for (std::size_t k = 0; k < a.size(); ++k) differ += !same(l[k], host_log(a[k]));
  for (std::size_t k = 0; k < ph.size(); ++k) {
    double hs, hc;
    host_sincos(ph[k], hs, hc);
    differ += !same(s[k], hs) + !same(c[k], hc);
  }
  for (std::size_t k = 0; k < turns.size(); ++k) {
    double hs, hc;
    host_turn(turns[k] >> 11, hs, hc);
    differ += !same(ts[k], hs) + !same(tc[k], hc);
  }
  const double el = log_error(log_arguments(), fetched(l, a.size())), er = root_error(x, fetched(r, x.size()));
  std::printf("log %.3f sqrt %.4f ulp; %lld values differ from the CPU's\n", el, er, differ);
  const bool ok = el <= kLogBound && er <= kRootBound && differ == 0;
  std::printf(ok ? "ok\n" : "FAILED\n");
  return ok ? 0 : 1;
}
