// Waits of the tcgen05 attention kernels, pair linears and matrix-memory segments that ran out (tc.cuh): the word they set in host memory, and the error that the next call makes of it.
#include "tc.cuh"

namespace b200 {

uint32_t* wait_status_word() {
  static uint32_t* const word = [] {   // pinned and mapped, at one address for every device; allocating it must not end a capture
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    void* p = nullptr;
    if (cudaHostAlloc(&p, 64, cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) *static_cast<volatile uint32_t*>(p) = 0;
    else p = nullptr, cudaGetLastError();
    cudaThreadExchangeStreamCaptureMode(&mode);
    return static_cast<uint32_t*>(p);
  }();
  return word;
}
int wait_status() {
  uint32_t* const w = wait_status_word();
  B200_REQUIRE(!w || __atomic_load_n(w, __ATOMIC_RELAXED) == 0 || __atomic_exchange_n(w, 0u, __ATOMIC_RELAXED) == 0, B200_ERR_CUDA,
               "a wait in a kernel of an earlier call ran out: that call's results are not valid");
  return B200_OK;
}

namespace {

// a barrier that nothing arrives at: the first wait runs out, the second finds the mark
__global__ void __launch_bounds__(64) expired_wait_kernel(uint32_t* status, int tries) {
  __shared__ uint64_t bar;
  __shared__ uint32_t mark;
  if (threadIdx.x == 0) {
    tc::mbar_init(&bar, 1);
    mark = 0;
  }
  __syncthreads();
  const tc::Waits wait(&mark, status, tries);
  wait(&bar, 0);
  wait(&bar, 0);
}

}  // namespace
}  // namespace b200

// debug helper (not in the public header): a kernel whose wait runs out after so many tries
extern "C" __attribute__((visibility("default"))) int b200_debug_expired_wait(int32_t tries, void* stream) {
  B200_CUDA(b200::launch(b200::expired_wait_kernel, dim3(1), dim3(64), (size_t)0, (cudaStream_t)stream, b200::wait_status_word(), tries));
  return B200_OK;
}
