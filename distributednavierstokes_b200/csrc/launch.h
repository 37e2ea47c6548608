// launch.h -- kernel launches shared by the library's translation units:
// the shared-memory opt-in per (device, kernel) and programmatic dependent
// launches.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <utility>

namespace dnsb {

// opt in to the dynamic shared memory a kernel launches with (needed whenever
// static + dynamic shared memory exceeds 48 KB; requested unconditionally).
// The attribute belongs to the kernel function (per device), not to the
// context, so contexts of different sizes in one process may only ever raise
// it: the largest request per (device, kernel) is kept.
inline cudaError_t raise_smem_of(int device, const void *kernel, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void *>, size_t> granted;
  std::lock_guard<std::mutex> lock(mu);
  size_t &cur = granted[{device, kernel}];
  if (bytes <= cur && cur != 0) return cudaSuccess;
  const size_t want = std::max(bytes, cur);
  const cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)want);
  if (e == cudaSuccess) cur = want;
  return e;
}

template <class K>
cudaError_t raise_smem(int device, K kernel, size_t bytes) {
  return raise_smem_of(device, reinterpret_cast<const void *>(kernel), bytes);
}

// Launch as a programmatic dependent of the stream's previous kernel: the
// grid may become resident while that kernel's last blocks run.  Only for
// kernels that execute pdl_wait() before any access to memory that an earlier
// kernel writes or reads (device_pdl.cuh).
template <class... P, class... A>
cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                             cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace dnsb
