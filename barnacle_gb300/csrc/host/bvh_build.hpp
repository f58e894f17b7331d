#pragma once
#include <cstdint>
#include <vector>

#include "../../../include/barnacle_gpu.h"
#include "host_math.hpp"

namespace bnh {
// Reference-compatible BVHNode.Build; see bvh_build.cpp.  Returns false when a leaf would hold
// more items than the reference's int8 count field.
bool bvh_build(const float* bounds, int32_t n, std::vector<bn_bvh_node>* nodes, std::vector<int32_t>* perm);
// whether the nodes fit a caller's array of 2 n (one for n = 0): boxes of infinite extent make chains of up
// to 129 nodes
inline bool fits_two_n(const std::vector<bn_bvh_node>& nodes, int32_t n) {
  return nodes.size() <= (n > 0 ? 2 * static_cast<size_t>(n) : 1);
}
}  // namespace bnh
