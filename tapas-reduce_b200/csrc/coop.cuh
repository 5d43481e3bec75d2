// Cooperative launches on a stream that may hold fewer blocks at once than the device.
#pragma once
#include <cuda_runtime.h>

namespace tb {

// Launches a cooperative kernel that is correct on any number of blocks: `launch(blocks)`
// is tried with half the blocks as long as it is refused as too large (the device's
// occupancy says nothing of a process's or a stream's share of the SMs).  blocks: in the
// most to try, out what was tried last.
template <class Launch>
inline cudaError_t launch_at_most(int &blocks, Launch launch) {
  for (;;) {
    const cudaError_t e = launch(blocks);
    if (e != cudaErrorCooperativeLaunchTooLarge || blocks <= 1) return e;
    cudaGetLastError();  // the refusal, which nothing else is to report
    blocks /= 2;
  }
}

}  // namespace tb
