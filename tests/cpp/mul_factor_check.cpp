// mul_f64 (fp64_int.cuh) with factors outside the normal range, bit for bit: half a time step
// below the smallest normal number is one of them.
#include "fp64_int.cuh"

#include <cmath>
#include <cstdio>
#include <random>

using namespace idpd;

int main() {
  std::mt19937_64 g(3);
  const double factors[] = {0.0, -0.0, 4.9e-324, 1e-310, 0x1.fffffffffffffp-1023, 2.3e-308, -1e-310,
                            -0.25, -1e300, INFINITY, -INFINITY, NAN, 1.7e308};
  const double edge[] = {0.0, -0.0, 1.0, -1.0, 128.0, -200.5, 1e300, 4.9e-324, INFINITY, -INFINITY, NAN};
  long bad = 0;
  for (double b : factors) {
    for (int k = 0; k < 100000; k++) {
      const uint64_t r = g();
      const double a = k < 11 ? edge[k]
                       : k % 2 ? f64_from(r)
                               : f64_from((r & ~(0x7ffull << 52)) | (1000ull + r % 60) << 52);
      const double got = mul_f64(a, b), want = a * b;
      if (f64_bits(got) != f64_bits(want) && !(std::isnan(got) && std::isnan(want)) && bad++ < 10)
        std::printf("%a * %a: %a, not %a\n", a, b, got, want);
    }
  }
  std::printf("%ld differences\n", bad);
  return bad ? 1 : 0;
}
