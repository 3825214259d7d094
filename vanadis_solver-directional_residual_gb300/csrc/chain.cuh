// chain.cuh -- short kernels that follow one another directly: the
// next one's blocks are brought up while the last ones of the one before are
// still running (programmatic dependent launch), instead of after them.
// Every kernel launched so begins with chain_wait, which returns when the
// kernel before is complete and what it wrote is visible; nothing is read
// before it, and what is read after it is read by plain loads: a read-only
// load (__ldg, const __restrict__) promises data that stays unchanged for the
// kernel's whole life, which begins while the kernel before still writes.
// It pays where a kernel takes about 10 us: the network's training pass (62
// launches) 859 -> 742 us, its forward pass 452 -> 425.  The Krylov iterations'
// kernels of 30 to 350 us, the block solve's among them, gained 0.3 per cent
// or lost 0.2, and stay plain.
#pragma once
#include <cuda_runtime.h>

namespace vdr {

__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... P, class... A>
cudaError_t chain_launch(void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t s,
                         const A &...args) {
  cudaLaunchAttribute after;
  after.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  after.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3((unsigned)block);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &after;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

}  // namespace vdr
