// launch.h -- kernel launches shared by the library's translation units:
// the shared-memory opt-in per (device, kernel) and programmatic dependent
// launches.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
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

template <class... P, class... A>
cudaError_t launch_as(bool dependent, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
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
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// SMs of the current device (148 where it cannot be told)
inline int sm_count() {
  static std::mutex mu;
  static std::map<int, int> known;
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  std::lock_guard<std::mutex> lock(mu);
  auto it = known.find(dev);
  if (it != known.end()) return it->second;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
    cudaGetLastError();
    return 148;
  }
  return known[dev] = n;
}

// Resident blocks of a kernel on the whole device (cached per device, kernel
// and launch shape).
inline long resident_blocks(const void *kernel, int threads, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, const void *, int, size_t>, long> known;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lock(mu);
  auto it = known.find({dev, kernel, threads, smem});
  if (it != known.end()) return it->second;
  int per = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;  // not known: an ordinary launch
  }
  return known[{dev, kernel, threads, smem}] = (long)per * sm_count();
}

// Launch of a kernel whose last argument says whether it is a programmatic
// dependent of the stream's previous kernel (pdl.cuh): where the grid is at
// most four waves.  A dependent grid's launch and prologue run under the
// previous kernel's tail (3 us per launch), but each block pays about 2 us in
// griddepcontrol.wait, the later waves' blocks too: 64^3 step 152 -> 116 us and
// 128^3 558 -> 526 with the rule; with every kernel dependent the 384 x 256 x
// 384 step went from 8.05 to 8.75 ms (the Crank-Nicolson solve, 62 waves,
// from 374 to 652 us).
constexpr int kDependentWaves = 4;
template <class K, class... A>
cudaError_t launch_pdl(K kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args) {
  const long blocks = (long)grid.x * grid.y * grid.z;
  const int dep = blocks <= kDependentWaves * resident_blocks(reinterpret_cast<const void *>(kernel),
                                                              (int)(block.x * block.y * block.z), smem);
  return launch_as(dep, kernel, grid, block, smem, stream, args..., dep);
}

}  // namespace dnsb
