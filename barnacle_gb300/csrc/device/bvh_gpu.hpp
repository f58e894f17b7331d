// Device side of the GPU BVH builder (k_bvh.cu): the reference-compatible binned SAH build of
// BVHNode.Build (Util/BVH.fs:99-247).  Ranges above kBvhSmall items are split level by level by
// kernels over all ranges of a level, smaller ones are finished by a warp each, and the preorder
// node array is assembled on the device.  The host (csrc/capi/bvh_gpu.cu) launches the levels and
// reads three counters after each.
#pragma once
#include <cuda_runtime.h>

#include "../../../include/barnacle_gpu.h"

namespace bn {

constexpr int kBvhBins = 12;
constexpr int kBvhSmall = 256;    // items of a range that one warp finishes
constexpr int kBvhMaxDepth = 64;

// one box to build over: (lo.xyz, item index as int bits), (hi.xyz, 0)
struct BvhItem {
  float4 a, b;
};

// A node above the small ranges: its range of items, what the level's kernels decide for it, its
// children (>= 0: top node; < 0: -(1 + small range)) and its place in the preorder.
struct BvhTop {
  float lo[3], hi[3];
  int first, last, depth;
  int axis, best;             // split axis; best SAH bin, or -1: median split
  float cmin, extent;
  float base;                 // count x area of the centroid bounds (the reference's cost offset)
  int chunk0;                 // the range's first 256-item chunk among the level's
  int left, right;
  int count, offset;          // nodes of the subtree, index of this node
};

// per-range reduction: box bounds and centroid bounds as order-preserving unsigned encodings,
// and per bound component the last item index whose coordinate is +-0 (the sign a sequential
// MinNative/MaxNative fold leaves on a zero bound)
struct BvhSegAcc {
  unsigned lo[3], hi[3], clo[3], chi[3];
  int zlo[3], zhi[3];
};

struct BvhBin {
  unsigned lo[3], hi[3];
  int cnt, pad;
};

// a range finished by one warp: its nodes (preorder, right child indices relative to the range's
// first node) go from nodes[2 * first] on
struct BvhSmallRange {
  int first, last, depth;
  int in_b;                   // the level's items are in buffer b
  int count, offset;
};

// device counters; flags: 1 a leaf over 127 items, 2 a NaN coordinate or centroid,
// 4 a range that outgrew its room.  n_chunks of the level; at the end the number of nodes
struct BvhCounters {
  int n_top, n_small, flags, n_chunks;
};

// all buffers of a build over n items
struct BvhBuffers {
  int n;
  BvhItem *a, *b;             // the items, level by level from one to the other
  BvhTop* top;                // n / 3 + 66 (a level has at most n / 257, 65 levels)
  BvhSmallRange* small;       // n / 3 + 67
  BvhSegAcc* acc;             // n / 257 + 1
  BvhBin* bins;               // 12 per range of a level
  int* chunk_cnt;             // 12 per chunk
  int* chunk_left;            // left items of the range before the chunk
  bn_bvh_node* nodes;         // nodes of the small ranges: 2 n + 160
  bn_bvh_node* out;           // the finished array: 2 n + 160
  int* perm;
  unsigned char* odd;         // per node of `out`: depth & 1, or null
  unsigned char* small_odd;   // the same for `nodes`
  BvhCounters* counters;
};

// first top node of each level; levels + 1 entries
struct BvhLevels {
  int levels;
  int first[kBvhMaxDepth + 2];
};

// items, counters and the root range (a top node, or a small range when n <= kBvhSmall)
cudaError_t bvh_launch_begin(const float* bounds, const BvhBuffers& w, cudaStream_t st);
// one level: top nodes [lb, le), their items from a (b if in_b) to the other buffer
cudaError_t bvh_launch_level(const BvhBuffers& w, int lb, int le, bool in_b, cudaStream_t st);
// the small ranges, then the node array: out, perm, and odd if it is not null
cudaError_t bvh_launch_finish(const BvhBuffers& w, const BvhLevels& lv, int n_small, cudaStream_t st);

}  // namespace bn
