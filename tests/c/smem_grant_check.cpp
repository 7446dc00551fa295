// allow_smem (csrc/smem_grant.h) against a fake runtime with two devices: prints
// what was asked for, "device:bytes".
#include <cstdio>

#include "smem_grant.h"

static int device = 0;
static bool refuse = false;

extern "C" cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int bytes) {
  if (refuse) return cudaErrorInvalidValue;
  printf("%d:%d ", device, bytes);
  return cudaSuccess;
}

static void kernel(int) {}

int main() {
  for (int launch = 0; launch < 4; launch++) {
    device = launch % 2;
    if (sns::allow_smem(kernel, 8 << 10, 200 << 10) != cudaSuccess) return 1;  // every block may have it
    if (sns::allow_smem(kernel, 60 << 10, 200 << 10) != cudaSuccess) return 2;
  }
  refuse = true;
  return sns::allow_smem(kernel, 60 << 10, 200 << 10) == cudaErrorInvalidValue ? 0 : 3;
}
