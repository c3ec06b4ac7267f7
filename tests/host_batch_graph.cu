// Host-side check of the graph length of a batch's two-pass step (no GPU
// needed): prints "ok" and exits 0, or the first failure and exits 1.
#include <cstdio>

#include "xfdtd_cuda_b200/csrc/handle.h"

int main() {
  for (int steps : {1, 7, 64, 1024})
    for (long long launches : {1LL, 2LL, 20LL, 63LL, 64LL, 65LL, 600LL, 2000LL, 4095LL, 4096LL, 4097LL, 20000LL}) {
      const long long n = batch_graph_steps(steps, launches);
      const bool fits = n * launches <= kBatchGraphLaunches || n == 1;
      const bool longest = n == steps || (n + 1) * launches > kBatchGraphLaunches;
      if (n < 1 || n > steps || !fits || !longest) {
        std::printf("FAIL %d steps at most, %lld launches a step: %lld steps\n", steps, launches, n);
        return 1;
      }
    }
  std::printf("ok\n");
  return 0;
}
