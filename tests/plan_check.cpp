// The plans of LPs whose vectors do not fit beside each other in shared memory (resident_plan.cuh): for each
// "m n" of the arguments, the blocks, the way the LP is solved and its shared memory. Read by
// tests/test_plan_cpu.py.
#include <cstdio>
#include <cstdlib>

#include "resident_plan.cuh"

int main(int argc, char** argv) {
  for (int k = 1; k + 1 < argc; k += 2) {
    const sih26::ResidentPlan pl = sih26::plan_outside(std::atoi(argv[k]), std::atoi(argv[k + 1]), 8);
    std::printf("%d %d %d\n", pl.cs, pl.outside, pl.bytes);
  }
  return 0;
}
