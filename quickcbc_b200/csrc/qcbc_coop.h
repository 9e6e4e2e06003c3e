// Cooperative launches of kernels whose result does not depend on the number of blocks.
#pragma once
#include <cuda_runtime.h>

namespace qcbc {

// launch(blocks) with as many blocks as the device takes at once, `most` at most.  A process may have fewer SMs
// than the device reports (a partition, or a share of them), and no query says so for every way of sharing; the
// launch does, without having run anything.  One block always fits.
template <class F>
cudaError_t launch_coop(int most, F launch) {
  for (int blocks = most;; blocks = (blocks + 1) / 2) {
    const cudaError_t e = launch(blocks);
    if (e != cudaErrorCooperativeLaunchTooLarge || blocks <= 1) return e;
    cudaGetLastError();                  // the refused launch's error is not the next call's
  }
}

}  // namespace qcbc
