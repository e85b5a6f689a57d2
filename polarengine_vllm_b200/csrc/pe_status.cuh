// Waits inside a kernel that ran out.  A kernel stores its code in the status word of its scratch; where a caller has no hold on
// that scratch (the host path's own buffers, a captured graph's pool) nobody could read it, so the code also goes to one word per
// device and source file, which pe_wait_status reads.  Included by the sources whose kernels wait.
#pragma once
#include "pe_common.cuh"

namespace pe {

static __device__ int g_wait_status;

// (a plain store: an atomic operation more made the matmul kernels spill, 40.2 -> 42.0 us over a layer's four launches)
__device__ __forceinline__ void record_timeout(int* status, int code) {
  if (status) atomicCAS(status, 0, code);
  asm volatile("st.volatile.global.s32 [%0], %1;" ::"l"(__cvta_generic_to_global(&g_wait_status)), "r"(code) : "memory");
}

// The word of this source file on the current device, once the stream has come so far.
#define PE_WAIT_STATUS_READER(name)                                                                       \
  int name(int clear, cudaStream_t st) {                                                                  \
    void* word = nullptr;                                                                                 \
    int v = 0;                                                                                            \
    PE_CUDA_TRY(cudaGetSymbolAddress(&word, g_wait_status));                                              \
    PE_CUDA_TRY(cudaMemcpyAsync(&v, word, sizeof(int), cudaMemcpyDeviceToHost, st));                      \
    PE_CUDA_TRY(cudaStreamSynchronize(st));                                                               \
    if (clear && v) PE_CUDA_TRY(cudaMemsetAsync(word, 0, sizeof(int), st));                               \
    return v;                                                                                             \
  }
int gemv_wait_status(int clear, cudaStream_t st);
int gemm_wait_status(int clear, cudaStream_t st);
int gemm_tmem_wait_status(int clear, cudaStream_t st);
int comm_wait_status(int clear, cudaStream_t st);

}  // namespace pe
