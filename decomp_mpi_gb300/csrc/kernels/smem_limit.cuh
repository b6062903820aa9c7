// The dynamic shared memory limit of a kernel function.
#pragma once
#include <cuda_runtime.h>

namespace {

// Opt-in shared memory of a block on sm_103a.
constexpr size_t SMEM_OPTIN = 232448;

// The limit is state of the function, shared by every plan and host thread:
// raised to the same value by every launch that needs more than the default
// 48 KB and never lowered, so that no thread takes it away between another
// one's call here and its launch.  fixed: the function's static shared
// memory at most.  (A launch that needs more than there is is refused here.)
template <typename K>
cudaError_t allow_smem(K kernel, size_t smem, size_t fixed = 0) {
  if (smem <= 48 * 1024) return cudaSuccess;
  const size_t most = SMEM_OPTIN - fixed;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(smem > most ? smem : most));
}

// Blocks per SM of a launch (0: it does not fit); CUDA's error where there is one.
template <typename K>
cudaError_t resident_blocks(K kernel, int threads, size_t smem, int *per_sm) {
  *per_sm = 0;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kernel, threads, smem);
}

}  // namespace
