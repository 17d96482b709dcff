// The constants of the flux's interface equilibrium (flux_core.cuh,
// flux_core32.cuh), host side.
//
// A node's equilibrium is evaluated in units of cd = c / 72, c = 1.5 s^2 / gamma
// (s the velocity unit: 1, or U in the FP32 deviation form), with k0 = 1 / c and
// k1 = 3 s / c. Every density at a face then carries the factor 72 cd k0 and
// every mass flux 24 cd k1 / s, both 1 up to the rounding of the constants. With
// each constant rounded by itself that is a common factor of all faces, up to
// 1 - 2^-53 at gamma = 1, and not a random error: so cd is taken within a few
// last places of c / 72, where k0 and k1, the nearest to 1 / (72 cd) and s / (24
// cd), leave both factors nearest to 1. Only the terms quadratic in the velocity
// see cd's own distance from c / 72 (`weight`: in FP64 they are a hundredth of the
// density's, in the deviation form as large as its own).
#pragma once

#include <cmath>

namespace plfbs {

template <typename T>
struct EqConstants {
  T k0, k1, cd;
};

template <typename T>
EqConstants<T> eq_constants(double gamma, double s, int places, double weight) {
  const long double c = 1.5L * (long double)s * s / gamma;
  const T mid = (T)(c / 72);
  EqConstants<T> best{};
  long double least = -1;
  for (int side = 0; side < 2; side++) {
    T cd = mid;
    for (int i = 0; i <= places; i++) {
      const T k0 = (T)(1 / (72 * (long double)cd)), k1 = (T)(s / (24 * (long double)cd));
      const long double e0 = 72 * (long double)cd * k0 - 1, e1 = 24 * (long double)cd * k1 / s - 1;
      const long double e2 = 72 * (long double)cd / c - 1;
      const long double e = e0 * e0 + e1 * e1 + weight * e2 * e2;
      if (least < 0 || e < least) {  // nearest to c / 72 first
        least = e;
        best = {k0, k1, cd};
      }
      cd = std::nextafter(cd, side ? (T)0 : (T)1e30);
    }
  }
  return best;
}

// The FP64 form's, and the deviation form's for the velocity unit U.
inline EqConstants<double> eq_constants64(double gamma) {
  return eq_constants<double>(gamma, 1.0, 8, 1e-4);
}
inline EqConstants<float> eq_constants32(double gamma, double U) {
  return eq_constants<float>(gamma, U, 2, 1.0);
}

}  // namespace plfbs
