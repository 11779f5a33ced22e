// Prints `registers computing-warpgroups fits` of the tensor-core kernels' register
// split (tc_core.cuh) and the two shares.
#include <stdio.h>

#include "tc_core.cuh"

int main() {
  printf("%d %d\n", scft::tc::kRegsCompute, scft::tc::kRegsIssue);
  for (int regs = 24; regs <= 255; ++regs)
    for (int c = 1; c <= 4; ++c) printf("%d %d %d\n", regs, c, scft::tc::split_fits(regs, c) ? 1 : 0);
  return 0;
}
