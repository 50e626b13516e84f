// Launches that overlap their set-up with the kernel before them in the stream
// (programmatic dependent launch).
#pragma once
#include <cuda_runtime.h>

#include "bt_common.cuh"

namespace bt {

// First statement of a kernel that launch_after starts.  Such a kernel, and every
// function that it calls, takes no __restrict__ pointers and makes no
// ld.global.nc loads: the compiler may move a load through a __restrict__
// parameter ahead of the wait (the memory clobber says nothing about it), and the
// non-coherent path is only for data that nothing writes while the kernel is
// there, which here is before its wait too.  (With them, a probe took its table's
// size from before the size was written.)  The loads with an L2 hint
// (bt_search.cuh) are asm without a memory clobber: their addresses have to come
// from something loaded after the wait.
__device__ __forceinline__ void after_previous() {
  dependents_may_launch();
  wait_for_previous();
}

// kernel<<<grid, block, smem, s>>>(args...) for a kernel that begins with
// after_previous().  A batch of the general path is a chain of some twenty short
// kernels with a launch gap of 1-2 us between them: a 2^21-request batch half
// INSERTs 475 -> 456 us, a 2^20-request STM batch 200 -> 191, 256 batches of
// 2^16 INSERTs 5,640 -> 5,420.
template <typename... Params, typename... Args>
inline void launch_after(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                         Args... args) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);  // errors: cudaGetLastError, as after <<< >>>
}

}  // namespace bt
