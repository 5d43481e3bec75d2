// launch_at_most against a stream that holds `room` blocks at once: what it tries, and
// what it reports.  usage: coop_launch_test; exit 0 when every check holds.
#include <cstdio>
#include <vector>

#include "coop.cuh"

static int failed = 0;
static void check(bool ok, const char *what) {
  if (!ok) {
    std::printf("failed: %s\n", what);
    failed = 1;
  }
}

int main() {
  for (int room : {0, 1, 2, 31, 32, 295, 296, 1000}) {
    for (int most : {1, 32, 296, 592}) {
      std::vector<int> tried;
      int blocks = most;
      const cudaError_t e = tb::launch_at_most(blocks, [&](int b) {
        tried.push_back(b);
        return b <= room ? cudaSuccess : cudaErrorCooperativeLaunchTooLarge;
      });
      check(tried.front() == most, "the most first");
      for (size_t i = 1; i < tried.size(); i++) check(tried[i] == tried[i - 1] / 2, "halved");
      check(tried.back() == blocks, "reports what it tried last");
      check(blocks >= 1, "never without a block");
      check((e == cudaSuccess) == (room >= 1), "succeeds where a block fits");
      check(e == cudaSuccess ? 2 * blocks > room || blocks == most : blocks == 1,
            "no smaller than it has to be");
    }
  }
  int blocks = 64, calls = 0;
  const cudaError_t e = tb::launch_at_most(blocks, [&](int) {
    calls++;
    return cudaErrorInvalidValue;
  });
  check(e == cudaErrorInvalidValue && calls == 1 && blocks == 64, "other errors at once");
  return failed;
}
