// TEST INFRASTRUCTURE: prints what gpq::laq_lanes, lsq_lanes and lhq_warp
// (gpupq_b200/csrc/phold_host.h) choose for each "<laq_mode> <num_lps> <events_per_lp>
// <lookahead>" line of stdin.
#include <cstdio>

#include "phold_host.h"

namespace gpq {
void set_last_error(const char*, ...) {}
}  // namespace gpq

int main() {
  gpq_phold_config c{};
  while (scanf("%u %u %u %f", &c.laq_mode, &c.num_lps, &c.events_per_lp, &c.lookahead) == 4)
    printf("%u %u %d\n", gpq::laq_lanes(c), gpq::lsq_lanes(c.num_lps), gpq::lhq_warp(c) ? 1 : 0);
  return 0;
}
