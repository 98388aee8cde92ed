// Correctly rounded operations of the stage update, for the device and (so
// that they can be checked against the host's own) the host.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define DGP_HD __host__ __device__ __forceinline__
#else
#define DGP_HD inline
#endif

namespace dgp {

// x / 3, rounded correctly: the product with the reciprocal, corrected by its
// exact remainder (Markstein 1990).  Where the remainder is zero (zeros of
// either sign among them) or not a number (infinities) the product stands.
DGP_HD double third(double x) {
  const double y = 1.0 / 3.0;
  const double q = x * y;
  const double r = fma(-3.0, q, x);
  return fabs(r) > 0.0 ? fma(r, y, q) : q;
}

}  // namespace dgp
