// The path-tracing megakernel (PathTracingIntegrator.Li): the work items of dev_mega.cuh on the
// path machine (dev_machine.cuh), and the chunk reduction shared by every integrator.
#define BN_COMPACT
#include <algorithm>

#include "dev_machine.cuh"
#include "dev_mega.cuh"

namespace bn {
namespace {

// The paths of the render's work items, item by item: a lane runs the samples of its item in
// order (acc is the plain loop's fma chain) and claims the next item from p.next.
template <bool kSimple>
struct MegaTask {
  const MegaParams& p;
  float inv_spp = 0.f;
  long long item = -1;
  int vi = 0, x = 0, y = 0, sid = 0, s1 = 0;
  V3 acc = {0.f, 0.f, 0.f};

  __device__ __forceinline__ explicit MegaTask(const MegaParams& q) : p(q) {
    inv_spp = __frcp_rn(static_cast<float>(q.spp));
  }

  __device__ __forceinline__ void finish(V3 L, IndepSampler&) {
    acc = fma3(mk(inv_spp, inv_spp, inv_spp), L, acc);
    if (++sid >= s1) p.partial[item] = make_float4(acc.x, acc.y, acc.z, 0.f);
  }

  __device__ __forceinline__ bool start(Ray* ray, IndepSampler* smp) {
    if (sid >= s1) {
      item = static_cast<long long>(claim_next(p.next));
      if (item >= p.n_items) return false;
      vi = find_view(p.item_offsets, p.n_views, item);
      const DevView& v = p.views[vi];
      const ItemPlace at = item_place(item - __ldg(&p.item_offsets[vi]), v.width, v.height);
      x = at.x;
      y = at.y;
      sid = at.chunk * p.spc;
      s1 = min(p.spp, sid + p.spc);
      acc = mk(0.f, 0.f, 0.f);
    }
    smp->state = xxhash32_three(static_cast<uint32_t>(x), static_cast<uint32_t>(y),
                                static_cast<uint32_t>(p.frame_id * p.spp + sid));
    const float upx = smp->next(), upy = smp->next();
    const float ulx = smp->next(), uly = smp->next();
    *ray = camera_ray<kSimple>(p.views[vi], x, y, upx, upy, ulx, uly);
    return true;
  }
};

template <bool kWT, int kWalk, bool kSimple>
__global__ void __launch_bounds__(kMachineThreads, kMachineBlocks)
    k_pt_machine(DevScene s, MegaParams p, int lanes) {
  MegaTask<kSimple> task(p);
  IndepSampler smp{0u};
  path_machine<kWT, kWalk, kSimple, false>(s, task, smp, p.max_depth, p.rr_depth, lanes);
}

// The chunk sums of renders whose paths ran in the wavefront: path_L holds the radiance of every
// path of pixels [first, first + n), samples of a pixel together.  One thread per chunk, the
// chunks of a pixel next to each other, so a warp reads one run of memory; the fma chain is the
// megakernel's, so the film is bit for bit the one it gives.
__global__ void __launch_bounds__(256) k_mega_chunks(MegaParams p, const float4* __restrict__ path_L, long long first,
                                                     unsigned n) {
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * static_cast<unsigned>(p.chunks)) return;
  const unsigned k = t / static_cast<unsigned>(p.chunks), c = t - k * static_cast<unsigned>(p.chunks);
  const long long gp = first + k;
  int vi = 0;
  while (vi + 1 < p.n_views && p.views[vi + 1].pixel_offset <= gp) ++vi;
  const DevView& v = p.views[vi];
  const int s0 = static_cast<int>(c) * p.spc, s1 = min(p.spp, s0 + p.spc);
  const float inv_spp = __frcp_rn(static_cast<float>(p.spp));
  const float4* L = path_L + static_cast<long long>(k) * p.spp;
  V3 acc = mk(0.f, 0.f, 0.f);
  for (int i = s0; i < s1; ++i) acc = fma3(mk(inv_spp, inv_spp, inv_spp), xyz(__ldcs(L + i)), acc);
  const long long npix = static_cast<long long>(v.width) * v.height;
  p.partial[__ldg(&p.item_offsets[vi]) + c * npix + (gp - v.pixel_offset)] = make_float4(acc.x, acc.y, acc.z, 0.f);
}

// one thread per pixel: sum the chunk partials in order, store at the flipped row (Film.fs:41-46)
__global__ void k_mega_reduce(MegaParams p) {
  const long long gp = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (gp >= p.n_pixels) return;
  int vi = 0;
  while (vi + 1 < p.n_views && p.views[vi + 1].pixel_offset <= gp) ++vi;
  const DevView& v = p.views[vi];
  const long long pix = gp - v.pixel_offset;
  const long long npix = static_cast<long long>(v.width) * v.height;
  const int x = static_cast<int>(pix % v.width), y = static_cast<int>(pix / v.width);
  const long long base = __ldg(&p.item_offsets[vi]) + pix;
  double r = 0.0, g = 0.0, b = 0.0;
  for (int c = 0; c < p.chunks; ++c) {
    const float4 q = p.partial[base + c * npix];
    r += q.x; g += q.y; b += q.z;
  }
  const long long out = v.pixel_offset + static_cast<long long>(v.height - y - 1) * v.width + x;
  p.film[3 * out] = static_cast<float>(r);
  p.film[3 * out + 1] = static_cast<float>(g);
  p.film[3 * out + 2] = static_cast<float>(b);
}

}  // namespace

cudaError_t launch_megakernel(const DevScene& s, const MegaParams& p, cudaStream_t st) {
  if (p.n_items <= 0) return cudaSuccess;
  if (p.integrator == BN_INTEGRATOR_NORMAL || p.integrator == BN_INTEGRATOR_DIRECT)
    return launch_megakernel_simple(s, p, st);
  if (p.count) {
    const long long grid = (p.n_items + 127) / 128;
    if (p.watertight) k_pt_mega<true, kWalkCount, BN_INTEGRATOR_PATH><<<grid, 128, 0, st>>>(s, p);
    else k_pt_mega<false, kWalkCount, BN_INTEGRATOR_PATH><<<grid, 128, 0, st>>>(s, p);
    return cudaGetLastError();
  }
  // Lambertian meshes walked binary, 8 K to 128 K paths: with a lane per path on less than two
  // rounds of warps, and walks of a few steps, the plain loop's lockstep costs less than the
  // machine's votes (Cornell box: 2,304 / 5,917 / 19,200 / 76,800 / 262,144 paths 0.180 0.193 0.182
  // 0.258 0.716 ms against 0.117 0.163 0.218 0.295 0.674)
  if (p.simple && !s.wide && p.n_paths >= 8192 && p.n_paths <= 131072) {
    const long long grid = (p.n_items + 127) / 128;
    if (p.watertight) k_pt_mega<true, kWalkBinary, BN_INTEGRATOR_PATH, true><<<grid, 128, 0, st>>>(s, p);
    else k_pt_mega<false, kWalkBinary, BN_INTEGRATOR_PATH, true><<<grid, 128, 0, st>>>(s, p);
    return cudaGetLastError();
  }
  // while (depth < maxDepth) never runs: every path's radiance is zero
  if (p.max_depth <= 0) return cudaMemsetAsync(p.partial, 0, static_cast<size_t>(p.n_items) * sizeof(float4), st);
  cudaError_t e = cudaMemsetAsync(p.next, 0, sizeof(*p.next), st);
  if (e != cudaSuccess) return e;
  auto run = [&](auto wt, auto walk, auto simple) {
    auto* k = k_pt_machine<decltype(wt)::value, decltype(walk)::value, decltype(simple)::value>;
    const int grid = static_cast<int>(std::min<long long>(p.n_items, resident_grid(k, kMachineThreads)));
    k<<<grid, kMachineThreads, 0, st>>>(s, p, machine_lanes(p.n_items, static_cast<long long>(grid) * (kMachineThreads / 32)));
  };
  using Yes = std::integral_constant<bool, true>;
  using No = std::integral_constant<bool, false>;
  dispatch_walk<false>(s, p.watertight, false, [&](auto wt, auto walk) {
    if constexpr (decltype(walk)::value == kWalkBinary) {
      // Lambertian meshes, uniform lights, pinhole views: the specialised path loop
      if (p.simple) return run(wt, walk, Yes{});
    }
    run(wt, walk, No{});
  });
  return cudaGetLastError();
}

cudaError_t launch_mega_chunks(const MegaParams& p, const float4* path_L, long long first, long long n, cudaStream_t st) {
  const long long threads = n * p.chunks;
  if (threads <= 0) return cudaSuccess;
  k_mega_chunks<<<static_cast<unsigned>((threads + 255) / 256), 256, 0, st>>>(p, path_L, first, static_cast<unsigned>(n));
  return cudaGetLastError();
}

cudaError_t launch_mega_reduce(const MegaParams& p, cudaStream_t st) {
  if (p.n_pixels <= 0) return cudaSuccess;
  k_mega_reduce<<<(p.n_pixels + 255) / 256, 256, 0, st>>>(p);
  return cudaGetLastError();
}

}  // namespace bn
