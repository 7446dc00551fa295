// Launches that are prepared while the kernel before them in their stream runs
// (programmatic dependent launch). A substage is a chain of short kernels, and
// between the end of one and the first instructions of the next an ordinary
// launch leaves ~3 us; with the dependence declared this way the next kernel's
// blocks come as the last block of the one before exits, and wait in
// chain_begin for its writes. Measured, us per step: parallel form 128 x 256
// 139 -> 118, 512 x 1024 294 -> 270; exact form 128 x 256 stretched 381 -> 344,
// 512 x 1024 660 -> 653.
//
// The blocks are not let in earlier (griddepcontrol.launch_dependents): those
// that wait fill whichever SMs have room at that time and leave the others with
// fewer, 512 x 1024 315 us per step. In the batched engine's graphs, whose
// launches are prepared ahead as it is, the gap is no shorter (222 us per step
// either way), so that its kernels are launched as before.
//
// No kernel launched this way reads through a const __restrict__ parameter or
// __ldg what another kernel of the chain writes: such loads could be moved in
// front of the wait.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace sns {

#ifdef __CUDACC__
// The first statement of every kernel launched this way, before any access to
// memory that a kernel writes: waits until the kernel before in the stream has
// ended and its writes are visible. A no-op in an ordinary launch.
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... P, typename... A>
cudaError_t chain_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
#endif

}  // namespace sns
