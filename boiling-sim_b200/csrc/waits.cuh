// waits.cuh -- words that kernels mark when a bounded wait gave up.  They lie in host
// memory that the device can write, so the host reads them without a synchronisation:
// the next call of the kind reports the error, and a caller that waits for its own call can
// ask at once (bsp_wait_status).
#pragma once
#include <cuda_runtime.h>

namespace bsp {

enum WaitKind { WAIT_SWEEPS = 0, WAIT_CONDUCTION = 1, WAIT_KINDS };

// Device address of a kind's word for the current device, or null.
int *wait_word(WaitKind kind);
// BSP_ERR_TIMEOUT if a wait of the kind gave up since the last call (which clears it).
int wait_status(WaitKind kind);

__device__ __forceinline__ void wait_gave_up(int *word) {
  *reinterpret_cast<volatile int *>(word) = 1;
  __threadfence_system();
}

}  // namespace bsp
