// cell_index (fp64_int.cuh) against the plain product, truncated and clamped to the grid,
// for coordinates inside the box, outside it and not numbers at all.
#include "fp64_int.cuh"

#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

using namespace idpd;

static int plain(double x, double inv_cs, int nc) {
  const double q = x * inv_cs;
  if (!(q > 0.0)) return 0;  // negative, zero, NaN
  return q >= (double)nc ? nc - 1 : (int)q;
}

int main() {
  std::mt19937_64 g(77);
  std::vector<double> edge = {0.0, -0.0, -4.9e-324, 4.9e-324, -1e-17, -0.3, -1.0, -7.5, -1e9, -3e9,
                              -1e30, -1e300, -1.7e308, 1e9, 2147483647.0, 2147483648.0, 3e9, 1e30,
                              1e300, 1.7e308, INFINITY, -INFINITY, NAN, -NAN};
  long bad = 0;
  const int cells[] = {1, 2, 3, 7, 64, 2048, 400000};
  for (int nc : cells) {
    for (int rep = 0; rep < 40; rep++) {
      const double side = nc * (1.0 + (double)(g() >> 11) * 0x1p-53 / nc);
      const double inv = (double)nc / side;
      std::vector<double> v = edge;
      for (double e : {0.0, side}) {
        v.push_back(e);
        v.push_back(std::nextafter(e, -1e9));
        v.push_back(std::nextafter(e, 1e9));
      }
      for (int c = 0; c <= nc && c < 200; c++) {
        v.push_back((double)c / inv);
        v.push_back(std::nextafter((double)c / inv, 0.0));
      }
      for (int k = 0; k < 2000; k++) {
        v.push_back((double)(g() >> 11) * 0x1p-53 * side);
        v.push_back(((double)(g() >> 11) * 0x1p-52 - 1.0) * 3.0 * side);
        v.push_back(f64_from(g()));  // any bits
      }
      for (double x : v) {
        const int c = cell_index(x, inv, nc);
        if ((c < 0 || c >= nc || c != plain(x, inv, nc)) && bad++ < 10)
          std::printf("cell_index(%a, %a, %d): %d, not %d\n", x, inv, nc, c, plain(x, inv, nc));
      }
    }
  }
  std::printf("%ld differences\n", bad);
  return bad ? 1 : 0;
}
