// cells_left and cells_right (cell_reach.hpp) for coordinates in their cell, where they are
// the plain expressions, and for any others, where they only have to be offsets of the stencil.
#include "cell_reach.hpp"

#include <cstdio>
#include <limits>
#include <random>

using namespace idpd;

int main() {
  std::mt19937 g(5);
  std::uniform_real_distribution<float> u(0.0f, 1.0f);
  long bad = 0;
  const float inf = std::numeric_limits<float>::infinity(), nan = std::nanf("");
  const float far[] = {1e6f, -1e6f, 3e9f, -3e9f, 1e20f, -1e20f, 3e38f, -3e38f, inf, -inf, nan, -nan};
  for (int k = 0; k < 400000; k++) {
    const int m = 2 + (int)(g() % 2), c0 = (int)(g() % (unsigned)(m - 1));
    const float side = (m == 2 ? 1.0f : 0.5f) * (1.0f + 0.33f * u(g)), inv = 1.0f / side;
    const float rem = 1.21f * u(g), x = ((float)c0 + u(g)) * side;
    const int l = cells_left(x, rem, inv, c0, m), r = cells_right(x, rem, inv, c0, m);
    int pl = c0 - (int)std::floor((x - rem) * inv), pr = (int)std::floor((x + rem) * inv) - c0;
    pl = pl > m ? m : (pl < 0 ? 0 : pl);
    pr = pr > m ? m : (pr < 0 ? 0 : pr);
    if ((l != pl || r != pr) && bad++ < 10)
      std::printf("x %a rem %a side %a: %d %d, not %d %d\n", x, rem, side, l, r, pl, pr);
    for (float f : {far[k % 12], x + 40.0f * (u(g) - 0.5f)}) {
      const int fl = cells_left(f, rem, inv, c0, m), fr = cells_right(f, rem, inv, c0, m);
      if ((fl < 0 || fl > m || fr < 0 || fr > m) && bad++ < 10)
        std::printf("x %a: %d %d\n", f, fl, fr);
    }
  }
  return bad ? 1 : 0;
}
