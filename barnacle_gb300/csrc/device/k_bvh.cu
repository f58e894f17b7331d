// GPU BVH builder kernels: the binned SAH build of BVHNode.Build (Util/BVH.fs:99-247) with the
// reference's results.
//
// Exactness.  Every float operation is written with _rn intrinsics in the reference's order (no
// contraction).  Bounds are reduced in any order, which gives the same value as the reference's
// sequential MinNative/MaxNative fold for boxes without NaN; the one thing an order-free reduction
// loses is the sign of a zero bound (the fold keeps the last item that compares equal), so where a
// bound is zero the last item with a zero coordinate gives its sign.  Centroid and bin bounds only
// feed differences and comparisons, where the sign of a zero does not matter.  The partition keeps
// the reference's order: items of bins <= best fill the range from the front in their order, the
// others from the back.  A split leaves no side empty unless the centroid extent is infinite, and
// then every range above is the whole input: the tree is a chain of 64 splits with an empty right
// side each, 129 nodes; any other tree over n items has at most 2 n - 1.
//
// Large ranges: a level is six launches over all its ranges (256-item chunks, one block each),
// whatever their number; decisions stay on the device.  Small ranges: a warp with the boxes in
// shared memory, permuting bytes.  400,000 boxes: 6.1 -> 0.25 ms for the small ranges (a thread each
// before), 2.6 -> 0.74 ms for the 14 levels (the host decided them), 3.3 -> 0.03 for the assembly.
// What is left is the levels' launches (each 2 to 15 us) and a synchronisation per level.
#include <math_constants.h>

#include <algorithm>
#include <cstdint>

#include "bvh_gpu.hpp"

namespace bn {
namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ unsigned f2o(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(unsigned o) {
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
__device__ __forceinline__ float cen(float lo, float hi) { return __fmul_rn(0.5f, __fadd_rn(lo, hi)); }
__device__ __forceinline__ float comp4(const float4& v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }

// bin = min(11, int(12 * (c - cmin) / extent))  (Util/BVH.fs:163-169)
__device__ __forceinline__ int bin_of(float c, float cmin, float extent) {
  const int k = __float2int_rz(__fdiv_rn(__fmul_rn(12.f, __fsub_rn(c, cmin)), extent));
  return k < kBvhBins - 1 ? k : kBvhBins - 1;
}
__device__ __forceinline__ int bin_of(const BvhItem& it, const BvhTop& t) {
  return bin_of(cen(comp4(it.a, t.axis), comp4(it.b, t.axis)), t.cmin, t.extent);
}

// 2 ((x y + y z) + z x) of a box's extent
__device__ __forceinline__ float area(const float lo[3], const float hi[3]) {
  const float x = __fsub_rn(hi[0], lo[0]), y = __fsub_rn(hi[1], lo[1]), z = __fsub_rn(hi[2], lo[2]);
  return __fmul_rn(2.f, __fadd_rn(__fadd_rn(__fmul_rn(x, y), __fmul_rn(y, z)), __fmul_rn(z, x)));
}

// the reference's split axis: the largest centroid extent, x before y before z
__device__ __forceinline__ int split_axis(float dx, float dy, float dz) {
  return (dx >= dy && dx >= dz) ? 0 : (dy >= dz ? 1 : 2);
}

// The cost of splitting after bin i (Util/BVH.fs:179-203): count x area of the bins up to i plus
// that of the others, plus the node's offset.  The reference adds the two terms from running unions
// in one loop; addition commutes, so each bin can be taken on its own.  Here lane i takes bin i (encoded)
// and a whole warp scans the unions from both ends; the lanes after the last split get infinity.  (With
// each lane running over all the bins by itself the small ranges of 400,000 boxes took 0.30 ms, now 0.25.)
__device__ __forceinline__ float split_cost(const BvhBin* bins, int lane, float base) {
  unsigned lo[2][3], hi[2][3];
  int cnt[2];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    lo[0][c] = lo[1][c] = lane < kBvhBins ? bins[lane].lo[c] : f2o(CUDART_INF_F);
    hi[0][c] = hi[1][c] = lane < kBvhBins ? bins[lane].hi[c] : f2o(-CUDART_INF_F);
  }
  cnt[0] = cnt[1] = lane < kBvhBins ? bins[lane].cnt : 0;
#pragma unroll
  for (int o = 1; o < kBvhBins; o <<= 1) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const unsigned l = __shfl_up_sync(kFull, lo[0][c], o), h = __shfl_up_sync(kFull, hi[0][c], o);
      if (lane >= o) {
        lo[0][c] = min(lo[0][c], l);
        hi[0][c] = max(hi[0][c], h);
      }
      lo[1][c] = min(lo[1][c], __shfl_down_sync(kFull, lo[1][c], o));
      hi[1][c] = max(hi[1][c], __shfl_down_sync(kFull, hi[1][c], o));
    }
    const int n = __shfl_up_sync(kFull, cnt[0], o);
    if (lane >= o) cnt[0] += n;
    // (lanes past the bins hold nothing, whatever they are given)
    const int m = __shfl_down_sync(kFull, cnt[1], o);
    if (lane + o < kBvhBins) cnt[1] += m;
  }
  float cost[2];
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    float l[3], h[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      l[c] = o2f(side ? __shfl_down_sync(kFull, lo[1][c], 1) : lo[0][c]);
      h[c] = o2f(side ? __shfl_down_sync(kFull, hi[1][c], 1) : hi[0][c]);
    }
    const int n = side ? __shfl_down_sync(kFull, cnt[1], 1) : cnt[0];
    cost[side] = __fmul_rn(static_cast<float>(n), area(l, h));
  }
  const float c = __fadd_rn(__fadd_rn(cost[0], cost[1]), base);
  return lane < kBvhBins - 1 ? (c == 0.f ? 0.f : c) : CUDART_INF_F;  // compared by their encodings: one zero
}

// ------------------------------------------------------------------ large ranges, level by level

__global__ void __launch_bounds__(256) k_bvh_begin(const float* __restrict__ bounds, BvhBuffers w) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    if (w.n > kBvhSmall) {
      w.top[0].first = 0;
      w.top[0].last = w.n;
      w.top[0].depth = 0;
    } else {
      w.small[0] = {0, w.n, 0, 0, 0, 0};
    }
  }
  bool nan = false;
  if (i < w.n) {
    float f[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      f[k] = bounds[6LL * i + k];
      nan |= f[k] != f[k];
    }
    // (a box from -inf to inf has no centroid either)
    for (int k = 0; k < 3; ++k) nan |= cen(f[k], f[3 + k]) != cen(f[k], f[3 + k]);
    w.a[i].a = make_float4(f[0], f[1], f[2], __int_as_float(i));
    w.a[i].b = make_float4(f[3], f[4], f[5], 0.f);
  }
  if (__any_sync(kFull, nan) && (threadIdx.x & 31) == 0) atomicOr(&w.counters->flags, 2);
}

// chunk numbers of the level's ranges (one block), and their accumulators cleared (the others)
__global__ void __launch_bounds__(1024) k_bvh_plan(BvhBuffers w, int lb, int le) {
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  if (blockIdx.x > 0) {
    for (int i = (blockIdx.x - 1) * 1024 + t; i < (le - lb) * kBvhBins; i += (gridDim.x - 1) * 1024) {
      BvhBin b;
      for (int k = 0; k < 3; ++k) {
        b.lo[k] = f2o(CUDART_INF_F);
        b.hi[k] = f2o(-CUDART_INF_F);
      }
      b.cnt = 0;
      b.pad = 0;
      w.bins[i] = b;
      if (i < le - lb) {
        BvhSegAcc a;
        for (int k = 0; k < 3; ++k) {
          a.lo[k] = a.clo[k] = f2o(CUDART_INF_F);
          a.hi[k] = a.chi[k] = f2o(-CUDART_INF_F);
          a.zlo[k] = a.zhi[k] = -1;
        }
        w.acc[i] = a;
      }
    }
    return;
  }
  __shared__ int warp_sum[32];
  __shared__ int carry;
  if (t == 0) carry = 0;
  __syncthreads();
  for (int s0 = lb; s0 < le; s0 += 1024) {
    const int s = s0 + t;
    const int c = s < le ? (w.top[s].last - w.top[s].first + 255) / 256 : 0;
    int x = c;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFull, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[wid] = x;
    __syncthreads();
    int before = carry;
    for (int k = 0; k < wid; ++k) before += warp_sum[k];
    if (s < le) w.top[s].chunk0 = before + x - c;
    __syncthreads();
    if (t == 1023) carry = before + x;
    __syncthreads();
  }
  if (t == 0) w.counters->n_chunks = carry;
}

// the range that holds chunk c, and the chunk's items
struct Chunk {
  int seg, begin, end;
};
__device__ __forceinline__ Chunk find_chunk(const BvhBuffers& w, int lb, int le, int c) {
  int lo = lb, hi = le - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (w.top[mid].chunk0 <= c) lo = mid;
    else hi = mid - 1;
  }
  const int begin = w.top[lo].first + (c - w.top[lo].chunk0) * 256;
  return {lo, begin, min(begin + 256, w.top[lo].last)};
}
// for every chunk of the level: f(chunk number, chunk), whole blocks
template <class F>
__device__ __forceinline__ void for_chunks(const BvhBuffers& w, int lb, int le, F f) {
  __shared__ Chunk shared_chunk;
  const int n = w.counters->n_chunks;
  for (int c = blockIdx.x; c < n; c += gridDim.x) {
    if (threadIdx.x == 0) shared_chunk = find_chunk(w, lb, le, c);
    __syncthreads();
    const Chunk ch = shared_chunk;
    f(c, ch);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) k_bvh_reduce(BvhBuffers w, const BvhItem* __restrict__ items, int lb, int le) {
  __shared__ unsigned s[12];
  __shared__ int z[6];
  const int t = threadIdx.x, lane = t & 31;
  for_chunks(w, lb, le, [&](int, const Chunk& c) {
    if (t < 12) s[t] = (t % 6) < 3 ? f2o(CUDART_INF_F) : f2o(-CUDART_INF_F);
    if (t < 6) z[t] = -1;
    __syncthreads();
    const int i = c.begin + t;
    const bool valid = i < c.end;
    float lo[3], hi[3];
    if (valid) {
      const BvhItem it = items[i];
      lo[0] = it.a.x; lo[1] = it.a.y; lo[2] = it.a.z;
      hi[0] = it.b.x; hi[1] = it.b.y; hi[2] = it.b.z;
    } else {
      lo[0] = lo[1] = lo[2] = CUDART_INF_F;
      hi[0] = hi[1] = hi[2] = -CUDART_INF_F;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const unsigned l = __reduce_min_sync(kFull, f2o(lo[k])), h = __reduce_max_sync(kFull, f2o(hi[k]));
      const float cc = cen(lo[k], hi[k]);
      const unsigned cl = __reduce_min_sync(kFull, valid ? f2o(cc) : kFull);
      const unsigned chh = __reduce_max_sync(kFull, valid ? f2o(cc) : 0u);
      const int zl = __reduce_max_sync(kFull, valid && lo[k] == 0.f ? i : -1);
      const int zh = __reduce_max_sync(kFull, valid && hi[k] == 0.f ? i : -1);
      if (lane == 0) {
        atomicMin(&s[k], l);
        atomicMax(&s[3 + k], h);
        atomicMin(&s[6 + k], cl);
        atomicMax(&s[9 + k], chh);
        atomicMax(&z[k], zl);
        atomicMax(&z[3 + k], zh);
      }
    }
    __syncthreads();
    BvhSegAcc* a = w.acc + (c.seg - lb);
    if (t < 3) {
      atomicMin(&a->lo[t], s[t]);
    } else if (t < 6) {
      atomicMax(&a->hi[t - 3], s[t]);
    } else if (t < 9) {
      atomicMin(&a->clo[t - 6], s[t]);
    } else if (t < 12) {
      atomicMax(&a->chi[t - 9], s[t]);
    } else if (t < 15) {
      if (z[t - 12] >= 0) atomicMax(&a->zlo[t - 12], z[t - 12]);
    } else if (t < 18) {
      if (z[t - 12] >= 0) atomicMax(&a->zhi[t - 15], z[t - 12]);
    }
  });
}

// per range: its box with the fold's zero signs, split axis and what the split needs
__global__ void __launch_bounds__(128) k_bvh_decide(BvhBuffers w, const BvhItem* __restrict__ items, int lb, int le) {
  const int s = lb + blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= le) return;
  const BvhSegAcc a = w.acc[s - lb];
  BvhTop* t = w.top + s;
  float clo[3], chi[3];
  for (int k = 0; k < 3; ++k) {
    float lo = o2f(a.lo[k]), hi = o2f(a.hi[k]);
    if (lo == 0.f && a.zlo[k] >= 0) lo = comp4(items[a.zlo[k]].a, k);
    if (hi == 0.f && a.zhi[k] >= 0) hi = comp4(items[a.zhi[k]].b, k);
    t->lo[k] = lo;
    t->hi[k] = hi;
    clo[k] = o2f(a.clo[k]);
    chi[k] = o2f(a.chi[k]);
  }
  // a range this long at the depth cap is a leaf of over 127 items
  if (t->depth >= kBvhMaxDepth) atomicOr(&w.counters->flags, 1);
  const float d[3] = {__fsub_rn(chi[0], clo[0]), __fsub_rn(chi[1], clo[1]), __fsub_rn(chi[2], clo[2])};
  const int axis = split_axis(d[0], d[1], d[2]);
  t->axis = axis;
  t->cmin = clo[axis];
  t->extent = d[axis];
  t->base = __fmul_rn(static_cast<float>(t->last - t->first), area(clo, chi));
  t->best = d[axis] == 0.f ? -1 : 0;
}

__global__ void __launch_bounds__(256) k_bvh_bins(BvhBuffers w, const BvhItem* __restrict__ items, int lb, int le) {
  __shared__ unsigned lo[kBvhBins][3], hi[kBvhBins][3];
  __shared__ int cnt[kBvhBins];
  const int t = threadIdx.x;
  for_chunks(w, lb, le, [&](int chunk, const Chunk& c) {
    const BvhTop h = w.top[c.seg];
    if (h.best < 0) return;
    if (t < kBvhBins * 3) {
      lo[t / 3][t % 3] = f2o(CUDART_INF_F);
      hi[t / 3][t % 3] = f2o(-CUDART_INF_F);
    }
    if (t < kBvhBins) cnt[t] = 0;
    __syncthreads();
    const int i = c.begin + t;
    if (i < c.end) {
      const BvhItem it = items[i];
      const int k = bin_of(it, h);
      atomicAdd(&cnt[k], 1);
      atomicMin(&lo[k][0], f2o(it.a.x));
      atomicMin(&lo[k][1], f2o(it.a.y));
      atomicMin(&lo[k][2], f2o(it.a.z));
      atomicMax(&hi[k][0], f2o(it.b.x));
      atomicMax(&hi[k][1], f2o(it.b.y));
      atomicMax(&hi[k][2], f2o(it.b.z));
    }
    __syncthreads();
    BvhBin* b = w.bins + kBvhBins * (c.seg - lb);
    if (t < kBvhBins * 3) {
      const int k = t / 3, a = t % 3;
      if (cnt[k]) {
        atomicMin(&b[k].lo[a], lo[k][a]);
        atomicMax(&b[k].hi[a], hi[k][a]);
      }
    } else if (t < kBvhBins * 4) {
      const int k = t - kBvhBins * 3;
      w.chunk_cnt[chunk * kBvhBins + k] = cnt[k];
      if (cnt[k]) atomicAdd(&b[k].cnt, cnt[k]);
    }
  });
}

// per range (a warp each): the cheapest bin, the two children, and the left items before each chunk
// A lane adds up four neighbouring chunks whose counts come in 16-byte loads, all in flight together: the
// first level's 1,563 chunks took 52 us one at a time (all levels together 0.21 ms, now 0.13).
constexpr int kChooseChunks = 4;
__global__ void __launch_bounds__(128) k_bvh_choose(BvhBuffers w, int lb, int le, int out_b) {
  const int lane = threadIdx.x & 31;
  const int s = lb + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (s >= le) return;
  BvhTop* t = w.top + s;
  const int first = t->first, last = t->last, count = last - first;
  int n_left, best = t->best;
  if (best < 0) {
    n_left = count / 2;
  } else {
    const BvhBin* bins = w.bins + kBvhBins * (s - lb);
    float c = split_cost(bins, lane, t->base);
    if (!(c < CUDART_INF_F)) c = CUDART_INF_F;  // a NaN cost is never the smallest
    const unsigned m = __reduce_min_sync(kFull, f2o(c));
    best = m == f2o(CUDART_INF_F) ? 0 : __ffs(__ballot_sync(kFull, f2o(c) == m)) - 1;
    n_left = __reduce_add_sync(kFull, lane <= best ? bins[lane].cnt : 0);
    int run = 0;
    const int nc = (count + 255) / 256;
    const int chunk0 = t->chunk0;
    for (int c0 = 0; c0 < nc; c0 += 32 * kChooseChunks) {
      int v[kChooseChunks], sum = 0;  // neighbouring chunks, their counts in flight together
#pragma unroll
      for (int j = 0; j < kChooseChunks; ++j) {
        const int ch = c0 + lane * kChooseChunks + j;
        v[j] = 0;
        if (ch < nc) {
          const int4* cnt = reinterpret_cast<const int4*>(w.chunk_cnt + (chunk0 + ch) * kBvhBins);
#pragma unroll
          for (int q = 0; q < kBvhBins / 4; ++q) {
            const int4 x = cnt[q];
            v[j] += (4 * q <= best ? x.x : 0) + (4 * q + 1 <= best ? x.y : 0) + (4 * q + 2 <= best ? x.z : 0) +
                    (4 * q + 3 <= best ? x.w : 0);
          }
        }
        sum += v[j];
      }
      int x = sum;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
      }
      int before = run + x - sum;
#pragma unroll
      for (int j = 0; j < kChooseChunks; ++j) {
        const int ch = c0 + lane * kChooseChunks + j;
        if (ch < nc) w.chunk_left[chunk0 + ch] = before;
        before += v[j];
      }
      run += __shfl_sync(kFull, x, 31);
    }
  }
  if (lane != 0) return;
  t->best = t->best < 0 ? -1 : best;
  const int split = first + n_left;
  auto child = [&](int f, int l) {
    if (l - f > kBvhSmall) {
      const int i = atomicAdd(&w.counters->n_top, 1);
      w.top[i].first = f;
      w.top[i].last = l;
      w.top[i].depth = t->depth + 1;
      return i;
    }
    const int i = atomicAdd(&w.counters->n_small, 1);
    w.small[i] = {f, l, t->depth + 1, out_b, 0, 0};
    return -1 - i;
  };
  // the arrays hold every child of ranges above 256 items down to the depth cap; a range at the
  // cap has raised the overflow flag and gets none
  if (t->depth >= kBvhMaxDepth) {
    t->left = t->right = 0;
    return;
  }
  t->left = child(first, split);
  t->right = child(split, last);
}

// items of bins <= best to first + (left items before them), the others to
// last - 1 - (right items before them): the reference's two-pointer fill.  A median split keeps its
// order.
__global__ void __launch_bounds__(256) k_bvh_partition(BvhBuffers w, const BvhItem* __restrict__ items,
                                                       BvhItem* __restrict__ out, int lb, int le) {
  __shared__ int warp_left[8];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  for_chunks(w, lb, le, [&](int chunk, const Chunk& c) {
    const BvhTop h = w.top[c.seg];
    const int i = c.begin + t;
    const bool valid = i < c.end;
    BvhItem it;
    bool left = false;
    if (valid) {
      it = items[i];
      left = h.best >= 0 && bin_of(it, h) <= h.best;
    }
    const unsigned m = __ballot_sync(kFull, left);
    if (lane == 0) warp_left[wid] = __popc(m);
    __syncthreads();
    if (!valid) return;
    int dst = i;
    if (h.best >= 0) {
      int lrank = w.chunk_left[chunk] + __popc(m & ((1u << lane) - 1u));  // left items before i in the range
      for (int k = 0; k < wid; ++k) lrank += warp_left[k];
      dst = left ? h.first + lrank : h.last - 1 - ((i - h.first) - lrank);
    }
    out[dst] = it;
  });
}

// ------------------------------------------------------------------ small ranges, a warp each

constexpr int kSmallWarps = 4;
constexpr int kFrames = 72;  // the depth cap of 64 bounds the stack
struct SmallShared {
  float box[6][kBvhSmall];       // lo.xyz, hi.xyz of the range's items, as they came
  unsigned char order[2][kBvhSmall];  // the items in their current order; the partition's other half
  BvhBin bins[kBvhBins];
  int2 stack[kFrames];           // first | last << 16, depth | parent << 8 (parent + 1; 0: none)
};

// The reference's recursion (Util/BVH.fs:99-237) over an explicit stack, nodes in preorder.
__global__ void __launch_bounds__(32 * kSmallWarps) k_bvh_small(BvhBuffers w, int n_small) {
  __shared__ SmallShared shared[kSmallWarps];
  const int lane = threadIdx.x & 31;
  const int si = blockIdx.x * kSmallWarps + (threadIdx.x >> 5);
  if (si >= n_small) return;
  SmallShared& sh = shared[threadIdx.x >> 5];
  const BvhSmallRange r = w.small[si];
  const BvhItem* items = r.in_b ? w.b : w.a;
  bn_bvh_node* out = w.nodes + 2LL * r.first;
  const int n = r.last - r.first;
  // room: 2 n nodes, or the whole array for the one range of a short input (the 129-node chain)
  const int room = w.n <= kBvhSmall ? 2 * w.n + 160 : 2 * n + 1;
  for (int i = lane; i < n; i += 32) {
    const BvhItem it = items[r.first + i];
    sh.box[0][i] = it.a.x; sh.box[1][i] = it.a.y; sh.box[2][i] = it.a.z;
    sh.box[3][i] = it.b.x; sh.box[4][i] = it.b.y; sh.box[5][i] = it.b.z;
    sh.order[0][i] = static_cast<unsigned char>(i);
  }
  int sp = 0, nn = 0;
  if (lane == 0) sh.stack[0] = make_int2(n << 16, r.depth);
  sp = 1;
  __syncwarp();
  while (sp > 0) {
    const int2 f = sh.stack[--sp];
    const int first = f.x & 0xffff, last = f.x >> 16, depth = f.y & 0xff, parent = (f.y >> 8) - 1;
    const int count = last - first;
    const int self = nn++;
    if (self >= room || sp + 2 > kFrames) {  // cannot happen (see the top of the file)
      if (lane == 0) atomicOr(&w.counters->flags, 4);
      return;
    }
    if (parent >= 0 && lane == 0) out[parent].right_or_offset = self;
    float lo[3] = {CUDART_INF_F, CUDART_INF_F, CUDART_INF_F}, hi[3] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
    float clo[3] = {CUDART_INF_F, CUDART_INF_F, CUDART_INF_F}, chi[3] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
    for (int i = first + lane; i < last; i += 32) {
      const int o = sh.order[0][i];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float l = sh.box[k][o], h = sh.box[3 + k][o], c = cen(l, h);
        lo[k] = fminf(lo[k], l);
        hi[k] = fmaxf(hi[k], h);
        clo[k] = fminf(clo[k], c);
        chi[k] = fmaxf(chi[k], c);
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      lo[k] = o2f(__reduce_min_sync(kFull, f2o(lo[k])));
      hi[k] = o2f(__reduce_max_sync(kFull, f2o(hi[k])));
      clo[k] = o2f(__reduce_min_sync(kFull, f2o(clo[k])));
      chi[k] = o2f(__reduce_max_sync(kFull, f2o(chi[k])));
    }
    if (lo[0] == 0.f || lo[1] == 0.f || lo[2] == 0.f || hi[0] == 0.f || hi[1] == 0.f || hi[2] == 0.f) {
      // a zero bound takes the sign of the last item with a zero coordinate
      int z[6] = {-1, -1, -1, -1, -1, -1};
      for (int i = first + lane; i < last; i += 32) {
        const int o = sh.order[0][i];
#pragma unroll
        for (int k = 0; k < 6; ++k)
          if (sh.box[k][o] == 0.f) z[k] = i;
      }
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const int at = __reduce_max_sync(kFull, z[k]);
        float* b = k < 3 ? &lo[k] : &hi[k - 3];
        if (*b == 0.f && at >= 0) *b = sh.box[k][sh.order[0][at]];
      }
    }
    const bool leaf = count <= 4 || depth >= kBvhMaxDepth;
    const float d[3] = {__fsub_rn(chi[0], clo[0]), __fsub_rn(chi[1], clo[1]), __fsub_rn(chi[2], clo[2])};
    const int axis = split_axis(d[0], d[1], d[2]);
    const float extent = axis == 0 ? d[0] : (axis == 1 ? d[1] : d[2]);
    if (lane == 0) {
      bn_bvh_node nd{};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        nd.bounds_min[k] = lo[k];
        nd.bounds_max[k] = hi[k];
      }
      if (leaf) {
        nd.right_or_offset = r.first + first;
        nd.is_leaf = 1;
        nd.count = static_cast<int8_t>(count);
        if (count > 127) atomicOr(&w.counters->flags, 1);
      } else {
        nd.split_axis = static_cast<int8_t>(axis);
        nd.right_or_offset = -1;  // set when the right child is emitted
      }
      out[self] = nd;
      if (w.odd) w.small_odd[2LL * r.first + self] = static_cast<unsigned char>(depth & 1);
    }
    if (leaf) continue;
    int split;
    if (extent == 0.f) {
      split = first + count / 2;
    } else {
      const float cmin = axis == 0 ? clo[0] : (axis == 1 ? clo[1] : clo[2]);
      if (lane < kBvhBins) {
        BvhBin b;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          b.lo[k] = f2o(CUDART_INF_F);
          b.hi[k] = f2o(-CUDART_INF_F);
        }
        b.cnt = 0;
        sh.bins[lane] = b;
      }
      __syncwarp();
      for (int i = first + lane; i < last; i += 32) {
        const int o = sh.order[0][i];
        const int k = bin_of(cen(sh.box[axis][o], sh.box[3 + axis][o]), cmin, extent);
        BvhBin* b = &sh.bins[k];
        atomicAdd(&b->cnt, 1);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          atomicMin(&b->lo[c], f2o(sh.box[c][o]));
          atomicMax(&b->hi[c], f2o(sh.box[3 + c][o]));
        }
      }
      __syncwarp();
      const float base = __fmul_rn(static_cast<float>(count), area(clo, chi));
      float c = split_cost(sh.bins, lane, base);
      if (!(c < CUDART_INF_F)) c = CUDART_INF_F;  // a NaN cost is never the smallest
      const unsigned m = __reduce_min_sync(kFull, f2o(c));
      const int best = m == f2o(CUDART_INF_F) ? 0 : __ffs(__ballot_sync(kFull, f2o(c) == m)) - 1;
      // the two-pointer fill, 32 items at a time into the other half, then back
      int nl = 0, nr = 0;
      for (int i0 = first; i0 < last; i0 += 32) {
        const int i = i0 + lane;
        const bool valid = i < last;
        const int o = valid ? sh.order[0][i] : 0;
        const bool left = valid && bin_of(cen(sh.box[axis][o], sh.box[3 + axis][o]), cmin, extent) <= best;
        const unsigned lm = __ballot_sync(kFull, left), rm = __ballot_sync(kFull, valid && !left);
        const unsigned below = (1u << lane) - 1u;
        if (left) sh.order[1][first + nl + __popc(lm & below)] = static_cast<unsigned char>(o);
        else if (valid) sh.order[1][last - 1 - nr - __popc(rm & below)] = static_cast<unsigned char>(o);
        nl += __popc(lm);
        nr += __popc(rm);
      }
      __syncwarp();
      for (int i = first + lane; i < last; i += 32) sh.order[0][i] = sh.order[1][i];
      split = first + nl;
    }
    if (lane == 0) {
      sh.stack[sp] = make_int2(split | (last << 16), (depth + 1) | ((self + 1) << 8));
      sh.stack[sp + 1] = make_int2(first | (split << 16), depth + 1);
    }
    sp += 2;
    __syncwarp();
  }
  if (lane == 0) w.small[si].count = nn;
  __syncwarp();
  for (int i = lane; i < n; i += 32) w.perm[r.first + i] = __float_as_int(items[r.first + sh.order[0][i]].a.w);
}

// ------------------------------------------------------------------ the preorder array

// Subtree sizes from the last level up, then node indices from the root down: a top node, its left
// subtree, its right subtree.  One block: the levels are short (a top node per 256 or more items).
__global__ void __launch_bounds__(1024) k_bvh_offsets(BvhBuffers w, BvhLevels lv) {
  auto count_of = [&](int ref) { return ref >= 0 ? w.top[ref].count : w.small[-1 - ref].count; };
  for (int l = lv.levels - 1; l >= 0; --l) {
    for (int i = lv.first[l] + threadIdx.x; i < lv.first[l + 1]; i += 1024)
      w.top[i].count = 1 + count_of(w.top[i].left) + count_of(w.top[i].right);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    w.top[0].offset = 0;
    w.counters->n_chunks = w.top[0].count;  // the number of nodes
  }
  __syncthreads();
  for (int l = 0; l < lv.levels; ++l) {
    for (int i = lv.first[l] + threadIdx.x; i < lv.first[l + 1]; i += 1024) {
      const BvhTop t = w.top[i];
      const int at_left = t.offset + 1, at_right = at_left + count_of(t.left);
      (t.left >= 0 ? w.top[t.left].offset : w.small[-1 - t.left].offset) = at_left;
      (t.right >= 0 ? w.top[t.right].offset : w.small[-1 - t.right].offset) = at_right;
    }
    __syncthreads();
  }
}

// a warp per small range and a lane per top node write the finished nodes
__global__ void __launch_bounds__(128) k_bvh_emit(BvhBuffers w, int n_top, int n_small) {
  const int lane = threadIdx.x & 31;
  const int wi = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (wi < n_small) {
    const BvhSmallRange r = w.small[wi];
    const int4* src = reinterpret_cast<const int4*>(w.nodes + 2LL * r.first);
    int4* dst = reinterpret_cast<int4*>(w.out + r.offset);
    for (int k = lane; k < 2 * r.count; k += 32) {
      int4 v = src[k];
      // second half: max.yz, link, (leaf, axis, count, mask); an interior node's link is relative
      if ((k & 1) && !(v.w & 0xff)) v.z += r.offset;
      dst[k] = v;
    }
    if (w.odd)
      for (int k = lane; k < r.count; k += 32) w.odd[r.offset + k] = w.small_odd[2LL * r.first + k];
    return;
  }
  const int i = (wi - n_small) * 32 + lane;
  if (i >= n_top) return;
  const BvhTop t = w.top[i];
  bn_bvh_node n{};
  for (int k = 0; k < 3; ++k) {
    n.bounds_min[k] = t.lo[k];
    n.bounds_max[k] = t.hi[k];
  }
  n.split_axis = static_cast<int8_t>(t.axis);
  n.right_or_offset = t.right >= 0 ? w.top[t.right].offset : w.small[-1 - t.right].offset;
  w.out[t.offset] = n;
  if (w.odd) w.odd[t.offset] = static_cast<unsigned char>(t.depth & 1);
}

// a short input's one range: its nodes are the array
__global__ void k_bvh_single(BvhBuffers w) {
  w.small[0].offset = 0;
  w.counters->n_chunks = w.small[0].count;
}

int blocks_for(long long n, int bs) { return static_cast<int>((n + bs - 1) / bs); }

}  // namespace

cudaError_t bvh_launch_begin(const float* bounds, const BvhBuffers& w, cudaStream_t st) {
  BvhCounters c{w.n > kBvhSmall ? 1 : 0, w.n > kBvhSmall ? 0 : 1, 0, 0};
  const cudaError_t e = cudaMemcpyAsync(w.counters, &c, sizeof(c), cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return e;
  k_bvh_begin<<<blocks_for(w.n, 256), 256, 0, st>>>(bounds, w);
  return cudaGetLastError();
}

cudaError_t bvh_launch_level(const BvhBuffers& w, int lb, int le, bool in_b, cudaStream_t st) {
  const BvhItem* in = in_b ? w.b : w.a;
  BvhItem* out = in_b ? w.a : w.b;
  const int ns = le - lb;
  // at most a partly filled chunk per range above the full ones
  const int chunks = std::min(w.n / 256 + ns, 152 * 16);
  k_bvh_plan<<<1 + std::min(blocks_for(ns * kBvhBins, 1024), 64), 1024, 0, st>>>(w, lb, le);
  k_bvh_reduce<<<chunks, 256, 0, st>>>(w, in, lb, le);
  k_bvh_decide<<<blocks_for(ns, 128), 128, 0, st>>>(w, in, lb, le);
  k_bvh_bins<<<chunks, 256, 0, st>>>(w, in, lb, le);
  k_bvh_choose<<<blocks_for(ns, 4), 128, 0, st>>>(w, lb, le, in_b ? 0 : 1);
  k_bvh_partition<<<chunks, 256, 0, st>>>(w, in, out, lb, le);
  return cudaGetLastError();
}

cudaError_t bvh_launch_finish(const BvhBuffers& w, const BvhLevels& lv, int n_small, cudaStream_t st) {
  k_bvh_small<<<blocks_for(n_small, kSmallWarps), 32 * kSmallWarps, 0, st>>>(w, n_small);
  const int n_top = lv.first[lv.levels];
  if (lv.levels > 0) k_bvh_offsets<<<1, 1024, 0, st>>>(w, lv);
  else k_bvh_single<<<1, 1, 0, st>>>(w);
  k_bvh_emit<<<blocks_for(n_small + blocks_for(n_top, 32), 4), 128, 0, st>>>(w, n_top, n_small);
  return cudaGetLastError();
}

}  // namespace bn
