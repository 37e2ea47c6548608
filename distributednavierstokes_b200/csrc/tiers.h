// tiers.h -- what the launches of the run-time-split kernels share (fftany.cu,
// spany.cu).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "fftany.cuh"

namespace dnsb {

constexpr size_t kSmemPerBlock = 110 * 1024;  // two blocks per SM at the least

// f(integral_constant<tier>)
template <class F>
cudaError_t by_tier(int tier, F f) {
  switch (tier) {
    case 10: return f(std::integral_constant<int, 10>());
    case 16: return f(std::integral_constant<int, 16>());
    case 25: return f(std::integral_constant<int, 25>());
    default: return cudaErrorInvalidValue;
  }
}

inline int threads_for(int items) { return std::min(FA_THREADS, std::max(32, (items + 31) / 32 * 32)); }

}  // namespace dnsb
