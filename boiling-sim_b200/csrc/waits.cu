// waits.cu -- host side of waits.cuh: one page of the library's own, mapped for every device.
#include "waits.cuh"

#include "bsp_common.cuh"

namespace bsp {

namespace {
alignas(4096) int g_words[1024];
}

int *wait_word(WaitKind kind) {
  void *d = nullptr;
  if (cudaHostGetDevicePointer(&d, g_words, 0) != cudaSuccess) {
    // first use, or the first after a device reset: allowed while a stream is captured too
    (void)cudaGetLastError();
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    cudaHostRegister(g_words, sizeof(g_words), cudaHostRegisterMapped | cudaHostRegisterPortable);
    (void)cudaGetLastError();  // another thread may have been first
    const cudaError_t e = cudaHostGetDevicePointer(&d, g_words, 0);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      return nullptr;
    }
  }
  return static_cast<int *>(d) + kind;
}

int wait_status(WaitKind kind) {
  if (__atomic_load_n(&g_words[kind], __ATOMIC_ACQUIRE) == 0) return BSP_OK;
  return __atomic_exchange_n(&g_words[kind], 0, __ATOMIC_ACQ_REL) ? BSP_ERR_TIMEOUT : BSP_OK;
}

}  // namespace bsp

extern "C" int bsp_wait_status(int kind) {
  if (kind < 0 || kind >= bsp::WAIT_KINDS) return BSP_ERR_ARG;
  return bsp::wait_status((bsp::WaitKind)kind);
}
