// Test infrastructure: csrc/eq_constants.hpp for tests/test_eq_constants.py.
#include "eq_constants.hpp"

extern "C" void eq64(double gamma, double out[3]) {
  const auto k = plfbs::eq_constants64(gamma);
  out[0] = k.k0, out[1] = k.k1, out[2] = k.cd;
}
extern "C" void eq32(double gamma, double U, float out[3]) {
  const auto k = plfbs::eq_constants32(gamma, U);
  out[0] = k.k0, out[1] = k.k1, out[2] = k.cd;
}
