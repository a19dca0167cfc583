// chained.cuh — launches that overlap the start of a kernel with the end of the one before it.
#pragma once

#include <cuda_runtime.h>

namespace lbm {

// Chained launches.  A kernel begins with chain_begin(): the next kernel of the stream, launched
// with launch_chained, may then be placed on the SMs as soon as every block here has started, and
// waits in its own chain_begin() until this one has completed and its writes are visible.  That
// hides the launch latency and the ramp between dependent kernels (B200, us per step: channel
// 96x48x48 11.4 -> 9.4, 192x96x96 TRT 60.4 -> 58.4, reference 480x240x4 26.8 -> 25.2).  Launched
// any other way, chain_begin() does nothing.
// A kernel that allocates tensor memory triggers after its allocation: a block of the next kernel
// that took the columns first would wait for this kernel, and this one for the columns.
// What the kernels before it wrote, a chained kernel reads with ordinary loads: it lives from
// before they end, and the read-only path (__ldg, const pointers declared __restrict__, which
// the compiler may load that way) is for data that nobody writes while a kernel lives.
__device__ __forceinline__ void chain_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_begin() {
  chain_trigger();
  chain_wait();
}

// Leaves a refused launch in the runtime's last error too, for callers that ask there.
template <class... P, class... A>
inline cudaError_t launch_chained_smem(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                       A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
// A launch that is refused is reported by the return value alone: the runtime's last error, which
// whoever launches next asks for, is taken back.
template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, A&&... args) {
  const cudaError_t e = launch_chained_smem(kernel, grid, block, 0, s, static_cast<A&&>(args)...);
  if (e != cudaSuccess) (void)cudaGetLastError();
  return e;
}

}  // namespace lbm
