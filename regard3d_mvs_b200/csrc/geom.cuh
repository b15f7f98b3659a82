// Double-precision 3-vector products of the multi-view kernels, in the
// left-to-right order ((a0 x + a1 y) + a2 z) that the reference's Eigen
// expressions evaluate for a fixed 3x3 matrix times a vector (and the
// library is built without contraction).
#pragma once

#include <cstring>

#include "simt.cuh"

namespace r3dgpu {

// Row i of a row-major 3x3 matrix times (x, y, z).
R3D_DEVICE double row3(const double* m, int i, double x, double y, double z) {
  return (m[3 * i] * x + m[3 * i + 1] * y) + m[3 * i + 2] * z;
}

// Row i of the transpose (column i) times (x, y, z).
R3D_DEVICE double col3(const double* m, int i, double x, double y, double z) {
  return (m[i] * x + m[3 + i] * y) + m[6 + i] * z;
}

// floor(q) as float and i = base + floor(q) for |q| < 2^22, without the
// conversion unit: adding 1.5 * 2^23 rounds to a whole number that the sum's
// low bits hold. Any other q (huge, infinite, NaN) gives some value of i; the
// integer arithmetic is modulo 2^32, so that callers may test q afterwards.
R3D_DEVICE float floor_small(float q, int base, int& i) {
  const float magic = 12582912.0F;
  const float t = __fadd_rn(q, magic);
  float r = __fsub_rn(t, magic);
  uint32_t bits, mbits;
  memcpy(&bits, &t, 4);
  memcpy(&mbits, &magic, 4);
  uint32_t k = static_cast<uint32_t>(base) + (bits - mbits);
  if (r > q) {
    r = __fsub_rn(r, 1.0F);
    --k;
  }
  i = static_cast<int>(k);
  return r;
}

}  // namespace r3dgpu
