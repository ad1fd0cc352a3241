// Kernels launched before the one in front of them on the stream has finished
// (programmatic dependent launch).
//
// A short kernel's launch, and the start of its blocks, take about as long as
// its work; launched this way they happen while the kernel in front drains.
// after_previous() holds every block until that kernel is complete and its
// writes are visible, so the order on the stream is what it was.
//
// Measured on a B200, one launch after the other against this: the cost
// model's 16 launches on 256 rows 227 -> 183 us, 15 per-operator calls over
// 600 MB 690 -> 663 us, 5 over 2 MiB 63 -> 58 us.
#pragma once

#include <cuda_runtime.h>

#include "device.h"

namespace bsz {

// First statement of a kernel launched by launch_after: waits for the work in
// front, then lets the next launch start its blocks as this grid's leave room.
// The pointers that the kernel reads through pass through the wait, so that no
// load, not even one marked read-only, can be moved in front of it.
template <class... P>
__device__ __forceinline__ void after_previous(P&... p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  (..., [&] { asm volatile("" : "+l"(p) :: "memory"); }());
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... K, class... A>
void launch_after(cudaStream_t stream, dim3 grid, dim3 block, size_t smem, void (*kernel)(K...), A... args) {
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = stream;
  c.attrs = &at;
  c.numAttrs = 1;
  BSZ_CUDA(cudaLaunchKernelEx(&c, kernel, static_cast<K>(args)...));
}

}  // namespace bsz
