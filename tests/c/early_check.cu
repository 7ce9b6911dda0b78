/* Prints, per shape, for launches of 1 to `wave` CTAs on 148 SMs, the ranges of
 * CTAs for which a stage does not let the next launch's CTAs in before its end
 * (host code; no device needed). */
#include "dg_mma.cuh"
#include "dg_stage.cuh"
#include "gpu_internal.h"

#include <cstdio>

using namespace bfam_b200;

static void show(const char *name, int per_sm, int late_from)
{
  StageParams sp{};
  sp.sms = 148;
  sp.slots = per_sm * sp.sms;
  int first = 0, last = 0, holes = 0;
  for (int n = 1; n <= 2 * sp.slots; ++n)
    if (!host::with_early(n, sp, late_from).early)
    {
      holes += first && last != n - 1;
      first = first ? first : n;
      last = n;
    }
  std::printf("%s %d %d %d %d\n", name, sp.slots, first, last, holes);
}

int main()
{
  show("node-3-fp64", 10, late_from<3, 3, double>());
  show("node-4-fp64", 6, late_from<3, 4, double>());
  show("node-5-fp64", 5, late_from<3, 5, double>());
  show("node-5-fp32", 4, late_from<3, 5, float>());
  show("node-2d-7", 8, late_from<2, 7, float>());
  show("mma-5", 5, mma_late_from<5>());
  show("mma-6", 3, mma_late_from<6>());
  show("mma-7", 2, mma_late_from<7>());
  show("node-7-fp32", 2, late_from<3, 7, float>());
  return 0;
}
