// Dynamic shared memory above the 48 KB that every block may have has to be
// asked for, per kernel and device.
#pragma once

#include <cstddef>

#include <cuda_runtime.h>

namespace sns {

// Before a launch with smem bytes of dynamic shared memory: `limit`, which is
// the same wherever the kernel is launched, so that threads that launch it with
// different sizes don't lower each other's. Asked for at each launch that may
// need it (the kernels' static arrays take up to 5 KB of the 48) and not once
// per process, since a second device has a grant of its own: no time shows it
// (64 x 128 through the calls 684.7 us before, 682.3 with it; 128 x 256
// parallel 2273 and 2280).
constexpr size_t kPlainSmem = 40 * 1024;
template <typename F>
cudaError_t allow_smem(F *kernel, size_t smem, size_t limit) {
  return smem <= kPlainSmem ? cudaSuccess
                            : cudaFuncSetAttribute(reinterpret_cast<const void *>(kernel),
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
}

}  // namespace sns
