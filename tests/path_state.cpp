// The wavefront's path state over a device whose allocations fail when told to: after any failure
// nothing is held, and a later call of any size gets every buffer again.
#include "../barnacle_gb300/csrc/capi/path_state.hpp"

#include <cstdio>
#include <cstdlib>
#include <map>

namespace {
std::map<void*, size_t> device;  // what is allocated
int fail_at = -1;                // allocations until one fails; -1: none does
}  // namespace

extern "C" cudaError_t cudaMalloc(void** p, size_t n) {
  if (fail_at >= 0 && fail_at-- == 0) return cudaErrorMemoryAllocation;
  *p = std::malloc(1);
  device[*p] = n;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void* p) {
  if (p && !device.erase(p)) std::abort();
  std::free(p);
  return cudaSuccess;
}

extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }

static size_t total() {
  size_t n = 0;
  for (auto& d : device) n += d.second;
  return n;
}
static void want(bool ok, const char* what, int k) {
  if (!ok) {
    std::printf("%s (failure at allocation %d)\n", what, k);
    std::exit(1);
  }
}
static void all_there(bnc::PathState& s, size_t pool, size_t paths, int k) {
  for (DevBuf* b : {&s.slot, &s.shadow, &s.q_bins, &s.q_active, &s.q_done, &s.q_key, &s.q_ray, &s.sh_key, &s.q_shadow})
    want(b->ptr && device.count(b->ptr) && b->bytes >= pool * sizeof(int), "a buffer is missing", k);
  want(s.slot.bytes >= 8 * pool * sizeof(float4) && s.shadow.bytes >= 4 * pool * sizeof(float4) &&
           s.q_bins.bytes >= bn::kNumBins * pool * sizeof(int),
       "a buffer is short", k);
  want(!paths || (s.path_L.ptr && s.path_L.bytes >= paths * sizeof(float4)), "no radiances", k);
  want(s.held() == total(), "held() differs from the device's count", k);
}

int main() {
  const size_t small = 1 << 20, large = 1 << 25;
  for (size_t paths : {size_t{0}, small})
    for (int k = 0; k < 10; ++k) {
      bnc::PathState s;
      want(s.reserve(small, paths) == cudaSuccess, "the first call failed", k);
      all_there(s, small, paths, k);
      fail_at = k;
      const bool failed = s.reserve(large, 2 * paths) == cudaErrorMemoryAllocation;
      want(failed == (k < (paths ? 10 : 9)), "a failed allocation was not reported", k);
      fail_at = -1;
      if (failed) want(total() == 0 && s.held() == 0, "memory kept after a failure", k);
      want(s.reserve(small, paths) == cudaSuccess, "the size that fitted before failed", k);
      all_there(s, small, paths, k);
      s.release();
      want(total() == 0, "memory kept after release", k);
    }
  bnc::PathState s;  // the limit: the bytes it counts are the bytes taken
  s.limit = small * bnc::PathState::bytes_per_slot() + 100 * sizeof(float4);
  want(s.reserve(small, 101) == cudaErrorMemoryAllocation && total() == 0, "the limit does not hold", -1);
  want(s.reserve(small, 100) == cudaSuccess && total() == s.limit, "the limit refuses what fits", -1);
  all_there(s, small, 100, -1);
  s.release();
  std::puts("ok");
}
