// Material data checks (host code only).
#pragma once

namespace e3d {

// Whether no strain has negative energy: from the bulk and shear modulus of an
// isotropic phase, from the constants of a cubic crystal (its bulk modulus is
// (c11 + 2 c12) / 3, its shear moduli (c11 - c12) / 2 and c44).  False for a NaN.
inline bool semidefinite(double bulk, double shear) { return bulk >= 0.0 && shear >= 0.0; }
inline bool semidefinite_cubic(double c11, double c12, double c44) {
  return c11 + 2.0 * c12 >= 0.0 && c11 >= c12 && c44 >= 0.0;
}

}  // namespace e3d
