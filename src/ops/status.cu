// Status words of the kernels whose waits are bounded: 0, or the role that gave up.  One of each kind per device, in the library's image: nothing is allocated at a
// kernel's first use, which may lie inside a caller's stream capture (an allocation or a copy on the default stream there ends the capture).
#include <atomic>
#include "ops_common.cuh"

namespace piccl_ops {

__device__ int g_status_words[kStatusKinds];

int* status_word(StatusKind kind) {
  static std::atomic<int*> known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  int* p = known[dev].load(std::memory_order_acquire);
  if (!p) {                           // may load the module: a capture in the default mode would refuse that
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    void* a = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&a, g_status_words);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) { cudaGetLastError(); return nullptr; }
    p = static_cast<int*>(a);
    known[dev].store(p, std::memory_order_release);
  }
  return p + kind;
}
int read_status(StatusKind kind) {
  const int* p = status_word(kind);
  int v = 0;
  if (p) cudaMemcpy(&v, p, sizeof v, cudaMemcpyDeviceToHost);
  return v;
}

}  // namespace piccl_ops

extern "C" {

// The words of the current device, out[0] GEMM, out[1] attention; clear: zero from now on.  A word stays set until it is cleared here.  Synchronises.
int piccl_ops_status(int* out, int clear) {
  int* p = piccl_ops::status_word(piccl_ops::STATUS_GEMM);
  if (!p) return -7;
  cudaError_t e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpy(out, p, piccl_ops::kStatusKinds * sizeof(int), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && clear) e = cudaMemset(p, 0, piccl_ops::kStatusKinds * sizeof(int));
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  return (int)e;
}
// Sets a word as a kernel that gave up would, for tests of what reads it.
int piccl_ops_test_set_status(int kind, int value) {
  if (kind < 0 || kind >= piccl_ops::kStatusKinds) return -1;
  int* p = piccl_ops::status_word((piccl_ops::StatusKind)kind);
  return p ? (int)cudaMemcpy(p, &value, sizeof value, cudaMemcpyHostToDevice) : -7;
}

}  // extern "C"
