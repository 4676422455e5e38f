// Compares fp64_int.cuh with the host's own FP64 arithmetic, bit for bit.
#include "fp64_int.cuh"

#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

using namespace idpd;

static long bad = 0;
static void same(double got, double want, const char* what, double a, double b) {
  if (f64_bits(got) != f64_bits(want) && !(std::isnan(got) && std::isnan(want)) && bad++ < 10)
    std::printf("%s(%a, %a): %a, not %a\n", what, a, b, got, want);
}

int main() {
  std::mt19937_64 g(20240607);
  std::vector<double> edge = {0.0, -0.0, 1.0, -1.0, 0.5, 2.0, 1.0 / 3.0, 4.9e-324, 2.3e-308, 1e-300,
                              1.7e308, INFINITY, -INFINITY, NAN, 0x1.fffffffffffffp0,
                              0x1.0000000000001p0, -0x1.fffffffffffffp52, 3.0e-39, 1.2e-38, 3.4e38,
                              0x1.000001p0, 0x1.000003p0, 0x1.fffffefffffffp-1, 0x1.ffffffp3};
  const std::vector<double> factors = {0.005, 0.0025, 0.01, 0x1.0000000000001p-8,
                                       0x1.fffffffffffffp-9, 1.0, 0.125, 1.1636363636363636,
                                       1.0 / 1.3, 64.0, 1e-300, 1e300};
  auto value = [&](int k) -> double {
    if (k < (int)edge.size()) return edge[k];
    const uint64_t b = g();
    switch (k % 5) {
      case 0: return f64_from(b);                                     // any bits
      case 1: return f64_from((b & ~(0x7ffull << 52)) | (1018ull + b % 12) << 52);
      case 2: return (double)(int64_t)(b >> 40) * 0x1p-20;             // few bits: ties
      case 3: return f64_from(((b & 0xffull) << 44) | (1020ull + b % 7) << 52);
      default: return std::ldexp((double)(int64_t)b, -60);
    }
  };
  for (int k = 0; k < 4000000; k++) {
    const double a = value(k), b = factors[(size_t)k % factors.size()];
    same(mul_f64(a, b), a * b, "mul", a, b);
    const double c = value((int)(g() % 4000000)) * (k & 8 ? 1.0 : 0x1p-9);
    same(add_f64(a, c), a + c, "add", a, c);
    same(add_f64(a, -a * (1.0 + 0x1p-52 * (double)(k & 3))), a - a * (1.0 + 0x1p-52 * (double)(k & 3)),
         "add", a, a);
    for (double z : edge) same(add_f64(a, z), a + z, "add", a, z);
    const float f = to_f32(a), w = (float)a;
    if (std::memcmp(&f, &w, 4) && !(std::isnan(f) && std::isnan(w)) && bad++ < 10)
      std::printf("to_f32(%a): %a, not %a\n", a, f, w);
    if (a >= 0.0 && a < 2147483648.0 && to_int(a) != (int)a && bad++ < 10)
      std::printf("to_int(%a): %d\n", a, to_int(a));
    if (std::isfinite(a) && abs_above(a, b) != (std::fabs(a) > b) && bad++ < 10)
      std::printf("abs_above(%a, %a)\n", a, b);
    if (std::isfinite(a) && in_fix(a) && to_fix(a) != (long long)std::trunc(a * 4294967296.0) &&
        bad++ < 10)
      std::printf("to_fix(%a): %lld\n", a, to_fix(a));
    const int n = (int)(g() % 4096);
    const double cs = 1.0 + (double)(g() >> 11) * 0x1p-53;
    same(mul_int_f64(n, cs), (double)n * cs, "mul_int", n, cs);
    const long long q = (long long)(g() >> (13 + k % 51)) * (g() & 1 ? -1 : 1);
    same(scale_force(q), (double)q / 67108864.0, "scale_force", (double)q, 0);
  }
  std::printf("%ld differences\n", bad);
  return bad ? 1 : 0;
}
