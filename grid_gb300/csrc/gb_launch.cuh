// gb_launch.cuh -- launches that overlap the end of the kernel before them (programmatic dependent
// launch).
//
// A solver is a chain of kernels of 3 to 200 us on one stream; between two of them the GPU idles
// 2 to 3 us (0.2 us inside a captured graph).  launch_pdl lets the next kernel's CTAs be placed, set
// up shared memory and read what no kernel in flight writes (links, neighbour tables: a gauge
// import ends with a stream synchronisation) as soon as the CTAs of the kernel before have
// ended, while its writes are still being flushed.  Every kernel launched this way calls pdl_wait() in
// every thread before its first other access to global memory: it returns when the kernel before
// has finished and its writes are visible.  A chain is ordered whole, because a kernel that
// waits finishes after the one it waited for.  Kernels, copies and events that are launched
// plainly wait as always.
//
// Measured, plain -> this: 8^4 CG 7.86 -> 5.90 ms, multishift solve 79 -> 63 ms, MpcDagMpc chain
// 24^4 x 12 1732 -> 1687 us.  With griddepcontrol.launch_dependents at the kernels' start, so that the
// next kernel's CTAs wait on the SMs beside the running ones, the same took 7.76 ms, 89 ms and
// 1918 us: it is not used.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace gb {

template <class... K, class... A>
inline cudaError_t launch_pdl(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = stream;
  c.attrs = &attr;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, static_cast<K>(std::forward<A>(args))...);
}

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// A pointer for use after pdl_wait(): loads through the read-only path (__ldg) carry no memory
// dependence, and this keeps the compiler from moving them before the wait.
template <class T> __device__ __forceinline__ T* after_wait(T* p) {
  asm volatile("" : "+l"(p)::"memory");
  return p;
}

}  // namespace gb
