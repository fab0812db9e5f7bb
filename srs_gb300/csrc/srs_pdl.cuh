// srs_pdl.cuh — launches whose start overlaps the end of the kernel before them.
//
// A step of the plain engines is a chain of short kernels.  With a full
// dependency the next one is launched when the last block of the one before has
// left: about 1.5 us without work on the device, and its parameters and constant
// data are then still to be fetched.  Launched with programmatic stream
// serialization it takes its places as they become free, reads what no step
// writes (geometry, channel elements), and waits for the one before it in
// pdl_wait.  Every thread of such a kernel calls pdl_wait before it touches
// anything that a step writes, so each kernel still sees all of the ones before.
// Measured: 64 steps of the allocation-free form (then one launch a step) 938 -> 765 us, a step of 32
// release sites (update, then gating) 250 -> 214 us, the adjoint of 64 steps over
// 8 x 69,696 elements 2.89 -> 2.30 ms.
#pragma once
#include <cuda_runtime.h>

namespace srs {

#ifdef __CUDACC__
// Waits until the kernel before this one has completed and its writes are visible.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next kernel take free places once every block of this one has called it.
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, args...);
}
#endif

}  // namespace srs
