// The wavefront's device memory that grows with its path slots.
#pragma once
#include <array>

#include "../device/wavefront.hpp"
#include "dev_buf.hpp"

namespace bnc {

struct PathState {
  DevBuf slot, q_active, q_bins, q_done, shadow, q_key, q_ray, sh_key, q_shadow;
  DevBuf path_L;  // radiance per path of a batch (ordered renders)
  size_t limit = 0;  // bytes that a call may ask for (bn_set_memory_limit; 0: what the GPU has)

  static constexpr size_t bytes_per_slot() { return 12 * sizeof(float4) + (bn::kNumBins + 6) * sizeof(int); }

  // `pool` slots and `paths` radiances.  Every buffer is looked at on every call, so that none is taken
  // for granted after an allocation failed, and what does not fit is given back whole: the caller goes
  // on without it, or with fewer slots.
  cudaError_t reserve(size_t pool, size_t paths) {
    const size_t bytes[] = {8 * pool * sizeof(float4), 4 * pool * sizeof(float4), bn::kNumBins * pool * sizeof(int),
                            paths * sizeof(float4), pool * sizeof(int)};  // of all(); the rest as the last
    cudaError_t e = limit && pool * bytes_per_slot() + paths * sizeof(float4) > limit ? cudaErrorMemoryAllocation : cudaSuccess;
    int k = 0;
    for (DevBuf* b : all()) {
      if (e == cudaSuccess) e = b->reserve(bytes[k < 4 ? k : 4]);
      ++k;
    }
    if (e != cudaSuccess) release();
    return e;
  }
  size_t held() {
    size_t n = 0;
    for (DevBuf* b : all()) n += b->bytes;
    return n;
  }
  void release() {
    for (DevBuf* b : all()) b->release();
  }

 private:
  std::array<DevBuf*, 10> all() {
    return {&slot, &shadow, &q_bins, &path_L, &q_active, &q_done, &q_key, &q_ray, &sh_key, &q_shadow};
  }
};

}  // namespace bnc
