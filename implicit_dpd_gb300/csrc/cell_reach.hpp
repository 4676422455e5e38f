// The cells of a row that come within a distance of a particle. Host and device code alike,
// compared with the plain expressions in the CPU tests.
#pragma once

#include <math.h>

#include "fp64_int.cuh"

namespace idpd {

// Cells to the left and to the right of search cell c0, at most m each, that come within rem
// of coordinate x (cells of side 1 / inv_side; x lies in c0). 0 for a coordinate that is no
// number or lies beyond the other side, as of a row outside the box, so that both are always
// offsets of the stencil.
IDPD_HD int cells_left(float x, float rem, float inv_side, int c0, int m) {
  return (int)fminf(fmaxf((float)c0 - floorf((x - rem) * inv_side), 0.0f), (float)m);
}
IDPD_HD int cells_right(float x, float rem, float inv_side, int c0, int m) {
  return (int)fminf(fmaxf(floorf((x + rem) * inv_side) - (float)c0, 0.0f), (float)m);
}

}  // namespace idpd
