// The plane grid of master_thesis_b200/csrc/plane_grid.h over many boxes, for tests/test_plane_grid.py.
#include "../../master_thesis_b200/csrc/plane_grid.h"

extern "C" {

// n nodes [lo, hi] on one axis with a child [clo, chi] each: the grid's origin, unit exponent and the
// child's two planes, as bytes and as the float levels that the traversal decodes from them.
void plane_grid_test(uint64_t n, const float* lo, const float* hi, const float* clo, const float* chi, float* origin,
                     int32_t* exponent, uint32_t* below, uint32_t* above, float* level_below, float* level_above) {
  for (uint64_t k = 0; k < n; ++k) {
    const swrx::PlaneGrid g = swrx::plane_grid(lo[k], hi[k]);
    origin[k] = g.origin;
    exponent[k] = (int32_t)g.ebyte - 127;
    below[k] = swrx::plane_below(g, clo[k]);
    above[k] = swrx::plane_above(g, chi[k]);
    level_below[k] = swrx::plane_level(below[k] << 16, 2);
    level_above[k] = swrx::plane_level(above[k] << 24, 3);
  }
}

}  // extern "C"
