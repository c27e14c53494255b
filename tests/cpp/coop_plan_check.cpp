// Prints the persistent cycle's plans for the devices and sizes on standard
// input: "launches sms smem N fp64 sweep2 m" -> "planned chunk grid fixed".
#include <cstdio>

#include "../../goal_gb300/csrc/coop_plan.h"

int main() {
  int launches, sms, smem, N, fp64, sweep2, m;
  while (std::scanf("%d %d %d %d %d %d %d", &launches, &sms, &smem, &N, &fp64, &sweep2, &m) == 7) {
    goal::CoopDevice d;
    d.launches = launches != 0;
    d.sms = sms;
    d.smem = smem;
    goal::CoopPlan p;
    const bool planned = goal::coop_plan(d, N, fp64 != 0, sweep2 != 0, p);
    std::printf("%d %d %d %zu\n", planned ? 1 : 0, p.chunk, p.grid,
                planned ? goal::coop_fixed_bytes(p.chunk, m, fp64 ? 8 : 4, sweep2 != 0) : 0);
  }
}
