// The grid of a wide node's child-box planes, shared by the host builder, the device builder, the
// refit and the traversal.
//
// A plane byte q stands for the float whose bits are 0x43000000 | q << 16, i.e. the levels 128, 129,
// .. 255 for q < 128 and 256, 258, .. 510 from there on: one byte permute on the integer pipe makes
// the byte a float. The integer-to-float conversion that a uniform 0..255 grid needs runs on the
// conversion pipe at 4 lanes per cycle and scheduler: the 48 planes of a node kept it busy for 384
// of about 500 issue cycles. The spacing doubles in the upper two thirds of the range, but 382 units
// span the node instead of 255, so the mean cell is the same (extent / 174 against extent / 181 over
// all extents; on the Cornell box, whose extents lie just above a power of two, 3.5 instead of 4.4
// triangle tests per ray). The level 128 of q = 0 is folded into the stored origin, which lies 128
// units below the node's lower corner. Measured with the traversal step as it is now, bounce
// traversal of the 2.4 M-triangle terrain image: 16.2 against 16.8 ms with the uniform grid on all
// axes (15.8 and 15.6 with it on one and two axes, where the Cornell renders lose 2-10 %), the
// bidirectional Cornell image 2.09 against 2.64 ms.
//
// The boxes stay conservative: planes are rounded outwards onto the levels, and the traversal's
// rounding of level * unit and origin (a few 2^-24 of the distance and of the node's extent) is far
// below the margin of extent / 65536 by which the builders enlarge every triangle box.
#pragma once

#include <math.h>
#include <stdint.h>

#include "swr_exact.cuh"

namespace swrx {

constexpr uint32_t kPlaneBits = 0x43000000u;

struct PlaneGrid {
  float origin;    // p: the plane of level v lies at p + v * unit
  uint32_t ebyte;  // the unit's biased exponent
  double per_unit;
};

SWR_HD double pow2(int e) {  // -1022 <= e <= 1023
#if defined(__CUDA_ARCH__)
  return __hiloint2double((e + 1023) << 20, 0);
#else
  const uint64_t b = (uint64_t)(e + 1023) << 52;
  double x;
  __builtin_memcpy(&x, &b, 8);
  return x;
#endif
}

// The grid of [lo, hi] on one axis: the smallest power-of-two unit whose levels 128..510, with an
// origin rounded down to a float, cover it.
SWR_HD PlaneGrid plane_grid(float lo, float hi) {
  const double cell = ((double)hi - (double)lo) * (1.0 / 382.0);
  // smallest ex with 2^ex >= cell
#if defined(__CUDA_ARCH__)
  const uint64_t b = (uint64_t)__double_as_longlong(cell);
#else
  uint64_t b;
  __builtin_memcpy(&b, &cell, 8);
#endif
  int ex = cell > 0.0 ? (int)((b >> 52) & 0x7FFu) - 1023 + ((b << 12) != 0 ? 1 : 0) : -126;
  ex = ex < -126 ? -126 : (ex > 127 ? 127 : ex);
  PlaneGrid g;
  for (;; ++ex) {
    const double at = (double)lo - 128.0 * pow2(ex);
    g.origin = (float)at;
    if ((double)g.origin > at) g.origin = nextafterf(g.origin, -INFINITY);
    // one step up at most, unless the box is far smaller than the float spacing at its position
    if (ex >= 127 || (double)g.origin + 510.0 * pow2(ex) >= (double)hi) break;
  }
  g.per_unit = pow2(-ex);
  g.ebyte = (uint32_t)(ex + 127);
  return g;
}

// The largest level at or below x, and the smallest at or above it, as plane bytes.
SWR_HD uint32_t plane_below(const PlaneGrid& g, float x) {
  const double v = ((double)x - (double)g.origin) * g.per_unit;
  const double q = v < 256.0 ? v - 128.0 : 128.0 + (v - 256.0) * 0.5;
  return (uint32_t)(q < 0.0 ? 0.0 : (q > 255.0 ? 255.0 : q));  // the conversion truncates
}
SWR_HD uint32_t plane_above(const PlaneGrid& g, float x) {
  const double v = ((double)x - (double)g.origin) * g.per_unit;
  const double q = v <= 255.0 ? v - 128.0 : 128.0 + (v <= 256.0 ? 0.0 : (v - 256.0) * 0.5);
  if (!(q > 0.0)) return 0u;
  if (q >= 255.0) return 255u;
  const uint32_t n = (uint32_t)q;
  return n + ((double)n < q ? 1u : 0u);
}

// Level of byte k (0..3) of w as a float: [0, 0, byte k, 0x43] from the low byte up.
SWR_HD float plane_level(uint32_t w, int k) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(__byte_perm(w, kPlaneBits, 0x7044u | ((uint32_t)k << 8)));
#else
  return bits2f(kPlaneBits | (((w >> (8 * k)) & 0xFFu) << 16));
#endif
}

}  // namespace swrx
