// Scene preparation on the device (scene_gpu.hpp).  Every float operation is the host preparation's,
// with _rn intrinsics, so the buffers are byte for byte the ones it makes (csrc/capi/scene_upload.cu).
//
// Each kernel reads and writes its arrays once.  The same loops on one host core, with the copies
// they needed, were 22 of the 28 ms in which the scene of 630,083 triangles was uploaded; it now takes
// 5.1 ms, most of it the builds (k_bvh.cu) and the copies of vertices and indices.
#include <cstdint>

#include "dev_geometry.cuh"
#include "scene_gpu.hpp"

namespace bn {
namespace {

struct Tri {
  V3 p0, p1, p2;
};
__device__ __forceinline__ Tri load_tri(const float* __restrict__ v, const int* __restrict__ idx, int t) {
  const long long a = 3LL * idx[3LL * t], b = 3LL * idx[3LL * t + 1], c = 3LL * idx[3LL * t + 2];
  return {mk(v[a], v[a + 1], v[a + 2]), mk(v[b], v[b + 1], v[b + 2]), mk(v[c], v[c + 1], v[c + 2])};
}

__global__ void __launch_bounds__(256) k_scene_boxes(const float* __restrict__ v, const int* __restrict__ idx, int n,
                                                     float* __restrict__ bounds) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const Tri q = load_tri(v, idx, t);
  const V3 lo = min_native(min_native(q.p0, q.p1), q.p2), hi = max_native(max_native(q.p0, q.p1), q.p2);
  float* b = bounds + 6LL * t;
  b[0] = lo.x; b[1] = lo.y; b[2] = lo.z;
  b[3] = hi.x; b[4] = hi.y; b[5] = hi.z;
}

__global__ void __launch_bounds__(256) k_scene_tris(const float* __restrict__ v, const int* __restrict__ idx,
                                                    const int* __restrict__ tri_material, const int* __restrict__ perm,
                                                    int n, float4* __restrict__ tris, float* __restrict__ areas) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int t = perm[k];
  const Tri q = load_tri(v, idx, t);
  float4* o = tris + 3LL * k;
  o[0] = make_float4(q.p0.x, q.p0.y, q.p0.z, __int_as_float(tri_material ? tri_material[t] : -1));
  o[1] = make_float4(q.p1.x, q.p1.y, q.p1.z, __int_as_float(t));
  o[2] = make_float4(q.p2.x, q.p2.y, q.p2.z, 0.f);
  areas[k] = __fmul_rn(0.5f, length(cross(sub(q.p1, q.p0), sub(q.p2, q.p0))));
}

__global__ void __launch_bounds__(256) k_scene_pdf(float* areas, int n, float sum) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) areas[k] = sum == 0.f ? __fdiv_rn(1.f, static_cast<float>(n)) : __fdiv_rn(areas[k], sum);
}

// a node: (min.xyz, max.x), (max.yz, link, bytes leaf | axis | count | mask)
struct Node {
  float lo[3], hi[3];
  int link;
  unsigned bytes;
  __device__ __forceinline__ bool leaf() const { return bytes & 0xffu; }
  __device__ __forceinline__ int axis() const { return static_cast<signed char>((bytes >> 8) & 0xffu); }
};
__device__ __forceinline__ Node get_node(const float4* __restrict__ nodes, int i) {
  const float4 a = nodes[2LL * i], b = nodes[2LL * i + 1];
  return {{a.x, a.y, a.z}, {a.w, b.x, b.y}, __float_as_int(b.z), static_cast<unsigned>(__float_as_int(b.w))};
}
// a record stands for an interior node two levels below another one's
__device__ __forceinline__ bool has_record(const WideParams& p, int i) {
  const unsigned bytes = static_cast<unsigned>(__float_as_int(p.nodes[2LL * (p.base + i) + 1].w));
  return !(bytes & 0xffu) && !p.odd[i];
}

__global__ void __launch_bounds__(1024) k_wide_rank(WideParams p) {
  __shared__ int warp_sum[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int i = blockIdx.x * 1024 + threadIdx.x;
  const bool rec = i < p.n && has_record(p, i);
  const unsigned m = __ballot_sync(0xffffffffu, rec);
  if (lane == 0) warp_sum[wid] = __popc(m);
  __syncthreads();
  int before = 0, total = 0;
  for (int k = 0; k < 32; ++k) {
    if (k < wid) before += warp_sum[k];
    total += warp_sum[k];
  }
  if (i < p.n) p.rank[i] = before + __popc(m & ((1u << lane) - 1u));
  if (threadIdx.x == 0) p.sums[blockIdx.x] = total;
}

// the blocks' sums to the records before each block, and after them the total (one block)
__global__ void __launch_bounds__(1024) k_wide_sums(int* sums, int n) {
  __shared__ int warp_sum[32];
  __shared__ int carry;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  if (t == 0) carry = 0;
  __syncthreads();
  for (int b0 = 0; b0 < n; b0 += 1024) {
    const int c = b0 + t < n ? sums[b0 + t] : 0;
    int x = c;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[wid] = x;
    __syncthreads();
    int before = carry;
    for (int k = 0; k < wid; ++k) before += warp_sum[k];
    if (b0 + t < n) sums[b0 + t] = before + x - c;
    __syncthreads();
    if (t == 1023) carry = before + x;
    __syncthreads();
  }
  if (t == 0) sums[n] = carry;
}

__device__ __forceinline__ int record_of(const WideParams& p, int i) {
  return p.first_record + p.sums[i >> 10] + p.rank[i];
}

__device__ __forceinline__ bool inside(const Node& in, const Node& outer) {
  bool ok = true;
  for (int a = 0; a < 3; ++a) ok = ok && outer.lo[a] <= in.lo[a] && in.hi[a] <= outer.hi[a];
  return ok;
}

// the record of node g: Collapse::emit of scene_upload.cu, whose preorder numbering is the rank
__global__ void __launch_bounds__(128) k_wide_fill(WideParams p) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < p.n_meshes) {
    const int r = p.mesh_base[i] - p.base;
    p.roots[i] = r < p.n && has_record(p, r) ? record_of(p, r) : -1;
  }
  if (i >= p.n || !has_record(p, i)) return;
  const int g = p.base + i;
  int m = 0, hi = p.n_meshes - 1;
  while (m < hi) {
    const int mid = (m + hi + 1) >> 1;
    if (p.mesh_base[mid] <= g) m = mid;
    else hi = mid - 1;
  }
  const int mb = p.mesh_base[m];
  const Node node = get_node(p.nodes, g);
  const int kids[2] = {g + 1, mb + node.link};
  int slot[4] = {-1, -1, -1, -1};
  int axis[3] = {node.axis(), 0, 0};
  bool nested = true;
  Node s[4];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const Node k = get_node(p.nodes, kids[c]);
    if (k.leaf()) {
      slot[2 * c] = kids[c];
      s[2 * c] = k;
    } else {
      slot[2 * c] = kids[c] + 1;
      slot[2 * c + 1] = mb + k.link;
      s[2 * c] = get_node(p.nodes, kids[c] + 1);
      s[2 * c + 1] = get_node(p.nodes, mb + k.link);
      axis[1 + c] = k.axis();
      nested = nested && inside(s[2 * c], k) && inside(s[2 * c + 1], k);
    }
  }
  if (!nested) atomicOr(p.flags, 1);
  float box[6][4];
  int ref[4] = {0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (slot[k] < 0 || (s[k].leaf() && ((s[k].bytes >> 16) & 0xffu) == 0)) {  // unused, or an empty leaf
#pragma unroll
      for (int r = 0; r < 6; ++r) box[r][k] = __int_as_float(0x7fc00000);
      continue;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      box[a][k] = s[k].lo[a];
      box[3 + a][k] = s[k].hi[a];
    }
    if (s[k].leaf()) {
      const int last = static_cast<int>((s[k].bytes >> 16) & 0xffu) - 1;
      if (last >= (1 << p.leaf_bits)) atomicOr(p.flags, 2);
      ref[k] = static_cast<int>(~((static_cast<unsigned>(s[k].link) << p.leaf_bits) | static_cast<unsigned>(last)));
    } else {
      ref[k] = record_of(p, slot[k] - p.base);
    }
  }
  // slot order per ray octant (bit a of the octant: d[a] > 0): the near child's pair first (left
  // when d[axis of g] > 0), each pair ordered by its child's split axis; 2 bits per slot
  unsigned orders[2] = {0u, 0u};
  for (int oct = 0; oct < 8; ++oct) {
    const bool lf = (oct >> (axis[0] & 3)) & 1;
    const bool fa = (oct >> (axis[lf ? 1 : 2] & 3)) & 1;
    const bool fb = (oct >> (axis[lf ? 2 : 1] & 3)) & 1;
    const int pa = lf ? 0 : 2, pb = 2 - pa;
    const unsigned v0 = pa + (fa ? 0 : 1), v1 = pa + (fa ? 1 : 0), v2 = pb + (fb ? 0 : 1), v3 = pb + (fb ? 1 : 0);
    orders[oct >> 2] |= (v0 | (v1 << 2) | (v2 << 4) | (v3 << 6)) << (8 * (oct & 3));
  }
  float4* o = p.records + 8LL * record_of(p, i);
#pragma unroll
  for (int k = 0; k < 6; ++k) o[k] = make_float4(box[k][0], box[k][1], box[k][2], box[k][3]);
  o[6] = make_float4(__int_as_float(ref[0]), __int_as_float(ref[1]), __int_as_float(ref[2]), __int_as_float(ref[3]));
  o[7] = make_float4(__uint_as_float(orders[0]), __uint_as_float(orders[1]), 0.f, 0.f);
}

unsigned blocks_for(long long n, int bs) { return static_cast<unsigned>((n + bs - 1) / bs); }

}  // namespace

cudaError_t scene_launch_boxes(const float* vertices, const int* indices, int n, float* bounds, cudaStream_t st) {
  if (n > 0) k_scene_boxes<<<blocks_for(n, 256), 256, 0, st>>>(vertices, indices, n, bounds);
  return cudaGetLastError();
}
cudaError_t scene_launch_tris(const float* vertices, const int* indices, const int* tri_material, const int* perm, int n,
                              float4* tris, float* areas, cudaStream_t st) {
  if (n > 0) k_scene_tris<<<blocks_for(n, 256), 256, 0, st>>>(vertices, indices, tri_material, perm, n, tris, areas);
  return cudaGetLastError();
}
cudaError_t scene_launch_pdf(float* areas, int n, float sum, cudaStream_t st) {
  if (n > 0) k_scene_pdf<<<blocks_for(n, 256), 256, 0, st>>>(areas, n, sum);
  return cudaGetLastError();
}
cudaError_t scene_launch_wide_count(const WideParams& p, cudaStream_t st) {
  const unsigned blocks = blocks_for(p.n, 1024);
  if (blocks) k_wide_rank<<<blocks, 1024, 0, st>>>(p);
  k_wide_sums<<<1, 1024, 0, st>>>(p.sums, static_cast<int>(blocks));
  return cudaGetLastError();
}
cudaError_t scene_launch_wide_fill(const WideParams& p, cudaStream_t st) {
  const int n = p.n > p.n_meshes ? p.n : p.n_meshes;
  if (n > 0) k_wide_fill<<<blocks_for(n, 128), 128, 0, st>>>(p);
  return cudaGetLastError();
}

}  // namespace bn
