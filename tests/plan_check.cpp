// The windows of LPs whose vectors do not fit in shared memory (resident_plan.cuh): for each "m n" of the
// arguments, the number of windows of x and of y. Read by tests/test_plan_cpu.py.
#include <cstdio>
#include <cstdlib>

#include "resident_plan.cuh"

int main(int argc, char** argv) {
  std::printf("%d\n", sih26::kWindow);
  for (int k = 1; k + 1 < argc; k += 2) {
    const sih26::ResidentPlan pl = sih26::plan_windows(std::atoi(argv[k]), std::atoi(argv[k + 1]), 1);
    std::printf("%d %d %d\n", pl.cs, pl.windows[0], pl.windows[1]);
  }
  return 0;
}
