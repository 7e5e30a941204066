// Host build of the key sort's choice of form (csrc/sort_rule.h).
#include "../../collisiondetection_gb300/csrc/sort_rule.h"

extern "C" int hc_sort_blocks(int64_t n, int cooperative, int sms, int per_sm) {
  return ccd::grid_sort_blocks(n, ccd::grid_sort_limit(cooperative != 0, sms, per_sm));
}
