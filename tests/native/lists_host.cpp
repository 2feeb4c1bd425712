// Test harness only: when the row product's lists make way for a plan (csrc/plan.h).
#include "plan.h"

extern "C" int pl_wants_lists(unsigned long long free, unsigned long long held, unsigned long long lists,
                              unsigned long long T, unsigned long long tb, unsigned long long budget) {
  return sfci::plan_wants_lists(free, held, lists, T, tb, budget) ? 1 : 0;
}
