// Query kernels: batched closest/any-hit tracing (the bit-exact parity path), batched BSDF
// eval/sample, and the hash-sampler stream.
#include <algorithm>

#include "dev_machine.cuh"
#include "launch.hpp"

namespace bn {
namespace {

__device__ __forceinline__ void warp_add_counters(DevCounters* c, unsigned long long rays, const TraceCounters& tc) {
  // warp-aggregated: one atomic per warp per counter
  for (int o = 16; o > 0; o >>= 1) {
    rays += __shfl_down_sync(0xffffffffu, rays, o);
  }
  unsigned long long nn = tc.nodes, tt = tc.tris, ii = tc.insts;
  for (int o = 16; o > 0; o >>= 1) {
    nn += __shfl_down_sync(0xffffffffu, nn, o);
    tt += __shfl_down_sync(0xffffffffu, tt, o);
    ii += __shfl_down_sync(0xffffffffu, ii, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&c->rays, rays);
    atomicAdd(&c->nodes, nn);
    atomicAdd(&c->tris, tt);
    atomicAdd(&c->insts, ii);
  }
}

__device__ __forceinline__ void put_closest(bn_hit* out, const DevScene& s, const Ray& ray, const HitRec& h) {
  const Interaction it = make_interaction(s, ray, h);
  out->t = h.t; out->u = it.u; out->v = it.v;
  out->instance = h.inst; out->primitive = h.tri;
  out->normal[0] = it.f.n.x; out->normal[1] = it.f.n.y; out->normal[2] = it.f.n.z;
  out->position[0] = it.p.x; out->position[1] = it.p.y; out->position[2] = it.p.z;
}

// one thread per ray: counting queries (the binary walk in the reference's order) and batches of
// about one ray per resident lane
template <bool kAny, bool kWT, int kWalk>
__global__ void __launch_bounds__(128) k_trace_plain(DevScene s, const bn_ray* __restrict__ rays, bn_hit* __restrict__ hits,
                                                     long long n, DevCounters* counters) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  TraceCounters tc{0, 0, 0};
  unsigned long long nr = 0;
  if (i < n) {
    const bn_ray r = rays[i];
    Ray ray;
    ray.o = mk(r.origin[0], r.origin[1], r.origin[2]);
    ray.d = mk(r.direction[0], r.direction[1], r.direction[2]);
    bn_hit out{};
    out.t = r.t_max;
    out.instance = out.primitive = -1;
    nr = 1;
    if (kAny) {
      if (trace_any<kWT, kWalk>(s, ray, r.t_max, &tc)) out.instance = 0;
    } else {
      HitRec h;
      if (trace_closest<kWT, kWalk>(s, ray, r.t_max, &h, &tc)) put_closest(&out, s, ray, h);
    }
    hits[i] = out;
  }
  if (kWalk == kWalkCount) warp_add_counters(counters, nr, tc);
}

// Persistent lanes: a lane whose walk has ended writes its hit and claims the next ray, together
// with its neighbours once half of the lanes still walk; the walking lanes vote on the kind of step
// (dev_machine.cuh).  1,000,003 closest hits in the instanced scene took 1.13 ms against 1.61 with a
// thread per ray, any hits 0.71 against 0.99, Cornell with objects 0.45 against 0.60; with the walk's
// later changes 0.97 and 0.62.  7 blocks per SM (72 registers); 8 blocks 0.99 ms, 6 blocks 1.00, 5 blocks
// 1.09; service when 20, 12 or 8 of 32 lanes still walk 1.13, 1.16, 1.19 ms where 16 took 1.13.  Few rays
// are spread over the warps, so none waits for a neighbour (64 rays of the Cornell box: 18 us against 27).
// Between the two, at about one ray per lane, the votes buy nothing (131,071 any hits in Cornell with
// objects, 131,071 and 65,537 closest hits among instances: 0.124, 0.276 and 0.258 ms against 0.101, 0.262
// and 0.240).
constexpr int kTraceBlocks = 7;
constexpr long long kTraceFew = 4096, kTraceMany = 196608;
template <bool kAny, bool kWT, int kWalk>
__global__ void __launch_bounds__(kMachineThreads, kTraceBlocks)
    k_trace(DevScene s, const bn_ray* __restrict__ rays, bn_hit* __restrict__ hits, long long n, unsigned long long* next,
            int lanes) {
  using Stack = std::conditional_t<kAny, SharedCodes<kMachineStack, kMachineThreads>,
                                   SharedStack<kMachineStack, kMachineThreads>>;
  __shared__ typename Stack::Entry stack_block[kMachineStack * kMachineThreads];
  Stack stk(stack_block);
  TraceCounters tc{0, 0, 0};
  Trav tr;
  tr.mode = kTravDone;
  int phase = static_cast<int>(threadIdx.x & 31) < lanes ? kLaneNew : kLaneIdle;
  long long at = 0;
  float tmax = 0.f;
  for (;;) {
    if (tr.mode == kTravDone && phase != kLaneIdle) {
      if (phase == kLaneClosest) {
        bn_hit out{};
        out.t = tmax;
        out.instance = out.primitive = -1;
        if (kAny) {
          if (tr.found()) out.instance = 0;
        } else if (tr.found()) {
          put_closest(&out, s, tr.wr, tr.hit());
        }
        hits[at] = out;
      }
      const unsigned long long i = claim_next(next);
      phase = i < static_cast<unsigned long long>(n) ? kLaneClosest : kLaneIdle;
      if (phase == kLaneClosest) {
        at = static_cast<long long>(i);
        const bn_ray r = rays[at];
        tmax = r.t_max;
        Ray ray;
        ray.o = mk(r.origin[0], r.origin[1], r.origin[2]);
        ray.d = mk(r.direction[0], r.direction[1], r.direction[2]);
        trav_init<kWalk>(tr, s, ray, tmax, &tc);
      }
    }
    const unsigned busy = __ballot_sync(0xffffffffu, phase != kLaneIdle);
    if (!busy) break;
    walk_down_to<kAny ? kAnyHit : kClosest, kWT, kWalk>(__popc(busy) / 2, tr, s, stk, &tc);
  }
}

template <bool kAny>
cudaError_t launch_trace_t(const DevScene& s, const bn_ray* rays, bn_hit* hits, long long n, unsigned flags,
                           unsigned long long* next, DevCounters* counters, cudaStream_t st) {
  if ((flags & BN_TRACE_COUNT) || (n > kTraceFew && n < kTraceMany)) {
    dispatch_walk<true>(s, flags & BN_TRACE_WATERTIGHT, flags & BN_TRACE_COUNT, [&](auto wt, auto walk) {
      k_trace_plain<kAny, decltype(wt)::value, decltype(walk)::value>
          <<<static_cast<unsigned>((n + 127) / 128), 128, 0, st>>>(s, rays, hits, n, counters);
    });
    return cudaGetLastError();
  }
  cudaError_t e = cudaMemsetAsync(next, 0, sizeof(*next), st);
  if (e != cudaSuccess) return e;
  dispatch_walk<false>(s, flags & BN_TRACE_WATERTIGHT, false, [&](auto wt, auto walk) {
    auto* k = k_trace<kAny, decltype(wt)::value, decltype(walk)::value>;
    const int grid = static_cast<int>(std::min<long long>(n, resident_grid(k, kMachineThreads)));
    k<<<grid, kMachineThreads, 0, st>>>(s, rays, hits, n, next,
                                        machine_lanes(n, static_cast<long long>(grid) * (kMachineThreads / 32)));
  });
  return cudaGetLastError();
}

__global__ void k_bsdf(DevScene s, const bn_bsdf_query* __restrict__ q, bn_bsdf_result* __restrict__ out, long long n,
                       bool sample) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const bn_bsdf_query a = q[i];
  bn_bsdf_result r{};
  if (a.material < 0 || a.material >= s.n_mats) {
    flag_error(s, BN_DEVERR_BAD_INDEX);
    out[i] = r;
    return;
  }
  const DevMaterial m = s.mats[a.material];
  const V3 wo = mk(a.wo[0], a.wo[1], a.wo[2]);
  if (sample) {
    const BsdfSample bs = bsdf_sample(m, wo, a.u_lobe, a.u_bsdf[0], a.u_bsdf[1]);
    r.bsdf[0] = bs.f.x; r.bsdf[1] = bs.f.y; r.bsdf[2] = bs.f.z; r.pdf = bs.pdf;
    r.wi[0] = bs.wi.x; r.wi[1] = bs.wi.y; r.wi[2] = bs.wi.z;
  } else {
    const BsdfEval e = bsdf_eval(m, wo, mk(a.wi[0], a.wi[1], a.wi[2]));
    r.bsdf[0] = e.f.x; r.bsdf[1] = e.f.y; r.bsdf[2] = e.f.z; r.pdf = e.pdf;
    r.wi[0] = a.wi[0]; r.wi[1] = a.wi[1]; r.wi[2] = a.wi[2];
  }
  out[i] = r;
}

__global__ void k_sampler_stream(const uint32_t* __restrict__ seeds, long long n_streams, int n_draws, float* __restrict__ out) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n_streams) return;
  IndepSampler smp{xxhash32_three(seeds[3 * i], seeds[3 * i + 1], seeds[3 * i + 2])};
  for (int k = 0; k < n_draws; ++k) out[i * n_draws + k] = smp.next();
}

}  // namespace

cudaError_t launch_trace(const DevScene& s, const bn_ray* rays, bn_hit* hits, long long n, unsigned flags,
                         unsigned long long* next, DevCounters* counters, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (flags & BN_TRACE_ANY) return launch_trace_t<true>(s, rays, hits, n, flags, next, counters, st);
  return launch_trace_t<false>(s, rays, hits, n, flags, next, counters, st);
}

cudaError_t launch_bsdf(const DevScene& s, const bn_bsdf_query* q, bn_bsdf_result* out, long long n, bool sample,
                        cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_bsdf<<<(n + 127) / 128, 128, 0, st>>>(s, q, out, n, sample);
  return cudaGetLastError();
}

cudaError_t launch_sampler_stream(const uint32_t* seeds, long long n_streams, int n_draws, float* out, cudaStream_t st) {
  if (n_streams <= 0) return cudaSuccess;
  k_sampler_stream<<<(n_streams + 127) / 128, 128, 0, st>>>(seeds, n_streams, n_draws, out);
  return cudaGetLastError();
}

}  // namespace bn
