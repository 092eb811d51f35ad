// Launches that overlap the end of the kernel ahead in the stream, and what such a kernel may do before it waits.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace q36 {

// Launch with programmatic stream serialisation: the grid may take its seats while the previous
// kernel in the stream drains.  The kernel must execute griddepcontrol.wait before it touches
// anything an earlier kernel may have written (and before it overwrites anything one may still read).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_after_previous(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem_bytes,
                                         cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Asks L2 for a piece of memory (16-byte aligned, a multiple of 16 bytes).  Reads nothing, so it may run before
// griddepcontrol.wait: a kernel that took its seat while the one ahead drains fills L2 with what it will need, whoever may
// still be writing some of it.
__device__ __forceinline__ void prefetch_l2(const void *p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// A contiguous span, a piece of 4 KB per thread: few requests, so that a kernel that is only seated for a microsecond gets
// them all out.
__device__ __forceinline__ void prefetch_l2_span(const uint8_t *p, uint32_t bytes, uint32_t thread) {
  constexpr uint32_t kPiece = 4096;
  if (thread < (bytes + kPiece - 1) / kPiece) prefetch_l2(p + thread * kPiece, min(kPiece, bytes - thread * kPiece));
}

}  // namespace q36
