// ql_rotation with a reciprocal root that is up to 2 ulp off (CUDA documents 1), over
// magnitudes and ratios. Prints the largest relative errors of the norm and of the two
// quotients, in units of 2^-53, and the number of wrong special values.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

namespace {
std::mt19937_64 g_rng(3);
double rsqrt(double x) {
  double r = static_cast<double>(1.0L / sqrtl(static_cast<long double>(x)));
  int64_t b;
  std::memcpy(&b, &r, 8);
  b += static_cast<int64_t>(g_rng() % 5) - 2;
  std::memcpy(&r, &b, 8);
  return r;
}
struct Idx {
  unsigned x = 0;
} threadIdx;
unsigned __ballot_sync(unsigned, bool p) { return p; }
void __syncwarp() {}
int __ffs(unsigned v) { return __builtin_ffs(static_cast<int>(v)); }
}  // namespace

#define __device__
#define __forceinline__ inline
#include QL_HEADER

int main() {
  const double u = std::ldexp(1.0, -53);
  std::normal_distribution<double> normal;
  std::uniform_real_distribution<double> range(-60.0, 60.0), spread(-12.0, 12.0);
  double worst_r = 0.0, worst_q = 0.0;
  for (int i = 0; i < 2000000; ++i) {
    const double scale = std::pow(10.0, range(g_rng));
    const double f = normal(g_rng) * scale, g = normal(g_rng) * scale * std::pow(10.0, spread(g_rng));
    double rr, s, c;
    ftlm::ql_rotation(f, g, rr, s, c);
    const long double r = hypotl(f, g);
    auto rel = [&](long double got, long double want) {
      return static_cast<double>(fabsl(got - want) / (fabsl(want) * u));
    };
    worst_r = std::fmax(worst_r, rel(rr, r));
    if (f != 0.0) worst_q = std::fmax(worst_q, rel(s, f / r));
    if (g != 0.0) worst_q = std::fmax(worst_q, rel(c, g / r));
  }
  int bad = 0;
  double rr, s, c;
  ftlm::ql_rotation(0.0, 0.0, rr, s, c);
  bad += rr != 0.0;
  ftlm::ql_rotation(3e-170, 4e-170, rr, s, c);  // the squares would underflow
  bad += std::fabs(rr - 5e-170) > 1e-185 || std::fabs(s - 0.6) > 1e-15 || std::fabs(c - 0.8) > 1e-15;
  ftlm::ql_rotation(3e200, 4e200, rr, s, c);  // and overflow
  bad += std::fabs(rr - 5e200) > 1e185 || std::fabs(s - 0.6) > 1e-15 || std::fabs(c - 0.8) > 1e-15;
  ftlm::ql_rotation(0.0, -2.0, rr, s, c);
  bad += rr != 2.0 || s != 0.0 || c != -1.0;
  std::printf("%.6f %.6f %d\n", worst_r, worst_q, bad);
  return 0;
}
