// Division by numbers known in advance: x / y from x (zh + zl), zh + zl = 1 / y
// (N. Brisebarre, J.-M. Muller, S. K. Raina, "Accelerating correctly rounded
// floating-point division when the divisor is known in advance", IEEE Trans.
// Computers 53, 2004).  The FP64 path divides by W_k and by 3 some 150 times per
// cell and step; two operations take the place of a division.
#pragma once

#include <cmath>

namespace ostc {

struct Reciprocal {
  double h, l;  // 1 / y = h + l, 0 < l <= ulp(h)
};

// h is 1 / y rounded down and never exact, so that l is positive: the two
// products of an infinite or a zero x then have the same sign.
inline Reciprocal reciprocal(double y) {
  double h = 1.0 / y;
  if (std::fma(-h, y, 1.0) <= 0) h = std::nextafter(h, 0.0);
  return {h, std::fma(-h, y, 1.0) / y};
}

// x / y.  Zeros keep their sign, infinities and NaN go through.  The quotient is
// the correctly rounded one where |x / y| >= 2^-960 (x zl does not underflow; the
// quotients near the middle of two doubles, which two operations could miss,
// are tested divisor by divisor); below, it may be the double beside it.
#ifdef __CUDACC__
__device__ __forceinline__ double div_by(double x, double zh, double zl) {
  return __fma_rn(x, zh, __dmul_rn(x, zl));
}
#else
inline double div_by(double x, double zh, double zl) { return std::fma(x, zh, x * zl); }
#endif

}  // namespace ostc
