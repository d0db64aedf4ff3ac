// px_units.h -- host conversions into the units of the integer pair sweeps
// (pair64.cu).  Plain C++: the same on every host.
#pragma once
#include <cmath>

// The squared cut-off of the long rows in units of r2, 2^(2 rho - 60) A^2.  r2
// is below 3 2^60; a cut-off beyond (1e300 without a skin) is none.  Compared
// before the conversion: of a number out of its range C++ defines no result,
// and x86-64 gives 0 for it where AArch64 gives the largest integer.
inline unsigned long long px_cut2(double rc2, int rho) {
  const double v = std::ldexp(rc2, 60 - 2 * rho);
  return v < 4611686018427387904.0 ? (unsigned long long)v : ~0ull;  // 2^62
}
