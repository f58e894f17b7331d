// GPU BVH builder, host side (kernels in k_bvh.cu): launches the levels of BVHNode.Build
// (Util/BVH.fs:99-247) over ranges above 256 items until none is left, reading three counters after
// each, then the small ranges and the assembly.  The result equals the host builder's
// (csrc/host/bvh_build.cpp) node for node and in the item permutation.  Boxes with a NaN
// coordinate or centroid, where the fold's order decides the bounds, are built by the host builder.
//
// The buffers (about 230 bytes per box) belong to the context and are kept from build to build up
// to 256 MB; larger ones are freed when the C call that needed them returns.
#include <algorithm>
#include <string>
#include <vector>

#include "../device/bvh_gpu.hpp"
#include "../host/bvh_build.hpp"
#include "context.hpp"

namespace bnc {

void BvhWork::release() {
  for (DevBuf* b : {&bounds, &items, &ranges, &level, &nodes, &out, &perm, &odd, &counters, &vertices, &indices, &slots,
                    &scene_odd, &wide}) b->release();
  if (host_counters) cudaFreeHost(host_counters);
  host_counters = nullptr;
}

void BvhWork::trim() {
  size_t total = 0;
  DevBuf* all[] = {&bounds, &items, &ranges, &level, &nodes, &out, &perm, &odd, &vertices, &indices, &slots, &scene_odd,
                   &wide};
  for (DevBuf* b : all) total += b->bytes;
  if (total > (256u << 20))
    for (DevBuf* b : all) b->release();
}

int gpu_bvh_build_resident(bn_context* ctx, const float* bounds_device, int32_t n, bool odd, bool* nan, int* n_nodes) {
  *nan = false;
  BvhWork& k = ctx->bvh;
  cudaStream_t st = ctx->stream;
  const size_t N = static_cast<size_t>(n), segs = N / 257 + 1, chunks = N / 256 + segs + 1, tops = N / 3 + 66;
  cudaError_t e;
  auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  const size_t top_b = up(tops * sizeof(bn::BvhTop)), small_b = up((tops + 1) * sizeof(bn::BvhSmallRange));
  const size_t acc_b = up(segs * sizeof(bn::BvhSegAcc)), bins_b = up(segs * bn::kBvhBins * sizeof(bn::BvhBin));
  const size_t cnt_b = up(chunks * bn::kBvhBins * sizeof(int));
  if ((e = ctx->reserve(k.items, 2 * N * sizeof(bn::BvhItem))) != cudaSuccess ||
      (e = ctx->reserve(k.ranges, top_b + small_b)) != cudaSuccess ||
      (e = ctx->reserve(k.level, acc_b + bins_b + cnt_b + chunks * sizeof(int))) != cudaSuccess ||
      (e = ctx->reserve(k.nodes, (2 * N + 160) * sizeof(bn_bvh_node))) != cudaSuccess ||
      (e = ctx->reserve(k.out, (2 * N + 160) * sizeof(bn_bvh_node))) != cudaSuccess ||
      (e = ctx->reserve(k.perm, N * sizeof(int))) != cudaSuccess ||
      (odd && (e = ctx->reserve(k.odd, 2 * (2 * N + 160))) != cudaSuccess) ||
      (e = ctx->reserve(k.counters, sizeof(bn::BvhCounters))) != cudaSuccess ||
      (!k.host_counters &&
       (e = cudaHostAlloc(&k.host_counters, sizeof(bn::BvhCounters), cudaHostAllocDefault)) != cudaSuccess))
    return ctx->cuda_fail(e, "BVH buffers");
  bn::BvhBuffers w{};
  w.n = n;
  w.a = k.items.as<bn::BvhItem>();
  w.b = w.a + N;
  w.top = k.ranges.as<bn::BvhTop>();
  w.small = reinterpret_cast<bn::BvhSmallRange*>(k.ranges.as<char>() + top_b);
  w.acc = k.level.as<bn::BvhSegAcc>();
  w.bins = reinterpret_cast<bn::BvhBin*>(k.level.as<char>() + acc_b);
  w.chunk_cnt = reinterpret_cast<int*>(k.level.as<char>() + acc_b + bins_b);
  w.chunk_left = reinterpret_cast<int*>(k.level.as<char>() + acc_b + bins_b + cnt_b);
  w.nodes = k.nodes.as<bn_bvh_node>();
  w.out = k.out.as<bn_bvh_node>();
  w.perm = k.perm.as<int>();
  w.odd = odd ? k.odd.as<unsigned char>() : nullptr;
  w.small_odd = odd ? w.odd + (2 * N + 160) : nullptr;
  w.counters = k.counters.as<bn::BvhCounters>();
  auto* c = static_cast<bn::BvhCounters*>(k.host_counters);
  auto sync = [&] {
    cudaError_t x = cudaMemcpyAsync(c, w.counters, sizeof(*c), cudaMemcpyDeviceToHost, st);
    return x == cudaSuccess ? cudaStreamSynchronize(st) : x;
  };
  if ((e = bn::bvh_launch_begin(bounds_device, w, st)) != cudaSuccess) return ctx->cuda_fail(e, "BVH items");
  bn::BvhLevels lv{};
  int n_small = n > bn::kBvhSmall ? 0 : 1, lb = 0, le = n > bn::kBvhSmall ? 1 : 0;
  bool in_b = false;
  while (lb < le && lv.levels <= bn::kBvhMaxDepth) {
    lv.first[lv.levels++] = lb;
    lv.first[lv.levels] = le;
    if ((e = bn::bvh_launch_level(w, lb, le, in_b, st)) != cudaSuccess || (e = sync()) != cudaSuccess)
      return ctx->cuda_fail(e, "BVH level");
    if (c->flags) break;
    n_small = c->n_small;
    lb = le;
    le = c->n_top;
    in_b = !in_b;
  }
  if (lv.levels == 0 || !c->flags) {
    if ((e = bn::bvh_launch_finish(w, lv, n_small, st)) != cudaSuccess || (e = sync()) != cudaSuccess)
      return ctx->cuda_fail(e, "BVH small ranges");
  }
  *nan = c->flags & 2;
  if (*nan) return BN_OK;
  if (c->flags & 1) return ctx->fail(BN_ERR_UNSUPPORTED, "BVH leaf larger than 127 items");
  if (c->flags) return ctx->fail(BN_ERR_UNSUPPORTED, "BVH build out of room");
  *n_nodes = c->n_chunks;
  return BN_OK;
}

int gpu_bvh_build(bn_context* ctx, const float* bounds, int32_t n, std::vector<bn_bvh_node>* nodes,
                  std::vector<int32_t>* perm) {
  bool nan = n <= 0;
  int n_nodes = 0;
  if (!nan) {
    cudaError_t e = ctx->reserve(ctx->bvh.bounds, 6 * static_cast<size_t>(n) * sizeof(float));
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(ctx->bvh.bounds.ptr, bounds, 6 * static_cast<size_t>(n) * sizeof(float), cudaMemcpyHostToDevice,
                          ctx->stream);
    if (e != cudaSuccess) return ctx->cuda_fail(e, "BVH bounds");
    const int rc = gpu_bvh_build_resident(ctx, ctx->bvh.bounds.as<float>(), n, false, &nan, &n_nodes);
    if (rc) return rc;
  }
  if (nan) {
    if (!bnh::bvh_build(bounds, n, nodes, perm)) return ctx->fail(BN_ERR_UNSUPPORTED, "BVH leaf larger than 127 items");
    return BN_OK;
  }
  nodes->resize(n_nodes);
  perm->resize(n);
  cudaMemcpyAsync(nodes->data(), ctx->bvh.out.ptr, nodes->size() * sizeof(bn_bvh_node), cudaMemcpyDeviceToHost, ctx->stream);
  cudaMemcpyAsync(perm->data(), ctx->bvh.perm.ptr, perm->size() * sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream);
  const cudaError_t e = cudaStreamSynchronize(ctx->stream);
  return e == cudaSuccess ? BN_OK : ctx->cuda_fail(e, "BVH download");
}

}  // namespace bnc

extern "C" int bn_bvh_build_device(bn_context* ctx, const float* bounds, int32_t n, bn_bvh_node* nodes,
                                   int32_t* n_nodes, int32_t* perm) {
  if (!ctx) return BN_ERR_INVALID_ARG;
  if ((!bounds && n > 0) || !nodes || !n_nodes || (!perm && n > 0) || n < 0)
    return ctx->fail(BN_ERR_INVALID_ARG, "bn_bvh_build_device: null pointer or negative count");
  cudaSetDevice(ctx->device);
  const bnc::TrimAtExit trim{ctx->bvh};
  cudaError_t e;
  bool nan = n == 0;
  int count = 0;
  if (n > 0) {
    const size_t bytes = 6 * static_cast<size_t>(n) * sizeof(float);
    if ((e = ctx->reserve(ctx->bvh.bounds, bytes)) != cudaSuccess ||
        (e = cudaMemcpyAsync(ctx->bvh.bounds.ptr, bounds, bytes, cudaMemcpyHostToDevice, ctx->stream)) != cudaSuccess)
      return ctx->cuda_fail(e, "BVH bounds");
    const int rc = bnc::gpu_bvh_build_resident(ctx, ctx->bvh.bounds.as<float>(), n, false, &nan, &count);
    if (rc) return rc;
  }
  if (nan) {
    std::vector<bn_bvh_node> nv;
    std::vector<int32_t> pv;
    if (!bnh::bvh_build(bounds, n, &nv, &pv)) return ctx->fail(BN_ERR_UNSUPPORTED, "BVH leaf larger than 127 items");
    if (!bnh::fits_two_n(nv, n)) return ctx->fail(BN_ERR_UNSUPPORTED, "BVH of more than 2 n nodes");
    std::copy(nv.begin(), nv.end(), nodes);
    *n_nodes = static_cast<int32_t>(nv.size());
    std::copy(pv.begin(), pv.end(), perm);
    return BN_OK;
  }
  // an infinite box makes a chain of 129 nodes: not into an array of 2 n
  if (count > 2 * static_cast<long long>(n)) return ctx->fail(BN_ERR_UNSUPPORTED, "BVH of more than 2 n nodes");
  // straight into the caller's arrays
  cudaMemcpyAsync(nodes, ctx->bvh.out.ptr, static_cast<size_t>(count) * sizeof(bn_bvh_node), cudaMemcpyDeviceToHost, ctx->stream);
  cudaMemcpyAsync(perm, ctx->bvh.perm.ptr, static_cast<size_t>(n) * sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream);
  if ((e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess) return ctx->cuda_fail(e, "BVH download");
  *n_nodes = count;
  return BN_OK;
}
