// Test infrastructure: csrc/march_rules.hpp for tests/test_march_rules.py.
#include "march_rules.hpp"

extern "C" int march_may_win(int compact, int fp32, int sms, int F) {
  return plfbs::march_may_win(compact, fp32, sms, F);
}
extern "C" int march_wins(int compact, int fp32, int n, int SF, int F) {
  return plfbs::march_wins(compact, fp32, n, SF, F);
}
