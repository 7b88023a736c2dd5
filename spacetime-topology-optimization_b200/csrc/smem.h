// The dynamic shared-memory ceiling of kernels that need more than 48 KB.
#pragma once

#include <mutex>

#include "errors.h"

namespace stt {

// Raises a kernel's ceiling to the device's opt-in maximum (less its static shared memory),
// once per device and kernel.  The ceiling belongs to the kernel, not to a call: set to each
// call's own size it would race between host threads, and a launch could meet another
// thread's smaller one and be refused.
template <auto Kernel>
int allow_smem() {
  static std::mutex mu;
  static bool done[64] = {};
  int dev = 0;
  STT_TRY(check_cuda(cudaGetDevice(&dev), "cudaGetDevice"));
  std::lock_guard<std::mutex> lock(mu);
  if (dev >= 0 && dev < 64 && done[dev]) return STT_OK;
  int optin = 0;
  cudaFuncAttributes fa;
  STT_TRY(check_cuda(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev), "smem attribute"));
  STT_TRY(check_cuda(cudaFuncGetAttributes(&fa, Kernel), "function attributes"));
  STT_TRY(check_cuda(cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          optin - (int)fa.sharedSizeBytes), "smem attr"));
  if (dev >= 0 && dev < 64) done[dev] = true;
  return STT_OK;
}

}  // namespace stt
