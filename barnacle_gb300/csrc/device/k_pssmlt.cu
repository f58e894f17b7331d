// Primary Sample Space Metropolis Light Transport (Extensions/Integrator/PSSMLT.fs).
//
//  k_mlt_bootstrap  BootstrapSingleChain (:247-273): the bootstrap paths, luminance y.
//                   A fresh MLTSampler's first iteration is a large step in which every
//                   dimension is drawn once from the inner sampler in order, so the bootstrap
//                   uses the inner sampler directly and stores no primary samples.
//  k_mlt_chains     RenderSingleChain (:275-377): a lane per chain, each at its own mutation and
//                   bounce.  The chain's primary samples live in HBM chain by chain as float4
//                   records (value, backup, last modification, backup of it): the seven draws of
//                   a bounce are 112 consecutive bytes whatever the neighbouring lanes do.
// Both run on the path machine (dev_machine.cuh).
// Kept from the reference: Reject restores every initialised dimension (:142-146); the
// acceptance min(1, y'/y) propagates NaN like MathF.Min; the chain's start is drawn from the
// AliasTable as built, which samples uniformly (Util/AliasTable.fs:20) unless the caller asks for
// the proportional table (BN_RENDER_FIXED_ALIAS).
#define BN_COMPACT
#include <algorithm>

#include "dev_machine.cuh"
#include "launch.hpp"
#include "mlt_sampler.cuh"
#include "pssmlt.hpp"

namespace bn {
namespace {

struct BootTask {
  const MltParams& p;
  int id = 0;
  __device__ __forceinline__ explicit BootTask(const MltParams& q) : p(q) {}
  __device__ __forceinline__ void finish(V3 L, IndepSampler&) { p.weights[id] = luminance(L); }
  __device__ __forceinline__ bool start(Ray* ray, IndepSampler* smp) {
    const unsigned long long i = claim_next(p.next);
    if (i >= static_cast<unsigned long long>(p.n_bootstrap)) return false;
    id = static_cast<int>(i);
    smp->state = xxhash32_two(static_cast<uint32_t>(p.frame_id), static_cast<uint32_t>(id));
    int x, y;
    *ray = mlt_camera(*p.view, *smp, &x, &y);
    return true;
  }
};

template <bool kWT, int kWalk>
__global__ void __launch_bounds__(kMachineThreads, kMachineBlocks) k_mlt_bootstrap(MltParams p, int lanes) {
  BootTask task(p);
  IndepSampler smp{0u};
  path_machine<kWT, kWalk, false, true>(p.scene, task, smp, p.max_depth, p.rr_depth, lanes);
}

__device__ __forceinline__ void splat(float* film, int pix, V3 c) {
  atomicAdd(film + 3LL * pix, c.x);
  atomicAdd(film + 3LL * pix + 1, c.y);
  atomicAdd(film + 3LL * pix + 2, c.z);
}

// The chain's state between its mutations, which only the Metropolis step touches: in shared
// memory, a column per thread, so that the walks keep their registers.
struct ChainState {
  V3 radiance, L;  // pending expected-value splat, radiance of the current state
  float y;         // its luminance
  int pix;         // its pixel
  int npix;        // pixel of the mutation in flight
  int it;          // mutation in flight; -1 = the chain's starting path
  int chain;       // -1 = none
  int bid;         // the bootstrap path the chain was drawn from
  uint32_t cs;     // the chain's sampler
};
constexpr int kChainWords = sizeof(ChainState) / 4;

struct MltTask {
  const MltParams& p;
  float* col;  // kChainWords columns of kMachineThreads
  unsigned long long accepted = 0;
  __device__ __forceinline__ MltTask(const MltParams& q, float* block) : p(q), col(block + threadIdx.x) {
    ChainState c{};
    c.chain = -1;
    put(c);
  }
  __device__ __forceinline__ ChainState get() const {
    union { ChainState c; float w[kChainWords]; } u;
#pragma unroll
    for (int k = 0; k < kChainWords; ++k) u.w[k] = col[k * kMachineThreads];
    return u.c;
  }
  __device__ __forceinline__ void put(const ChainState& c) {
    union { ChainState c; float w[kChainWords]; } u;
    u.c = c;
#pragma unroll
    for (int k = 0; k < kChainWords; ++k) col[k * kMachineThreads] = u.w[k];
  }

  // the Metropolis step of the path that ended
  __device__ __forceinline__ void finish(V3 Ln, MltSampler& m) {
    ChainState c = get();
    const float yn = luminance(Ln);
    if (c.it < 0) {
      c.L = Ln;
      c.y = yn;
      m.accept();
      m.inner = xxhash32_three(static_cast<uint32_t>(c.chain), static_cast<uint32_t>(c.bid),
                               static_cast<uint32_t>(p.frame_id));
      c.pix = c.npix;
    } else {
      const float inv_b = __frcp_rn(p.b);
      const float ratio = __fdiv_rn(yn, c.y);
      const float acc = ratio != ratio ? ratio : fminf(1.f, ratio);  // MathF.Min propagates NaN
      const float w_old = __fdiv_rn(__fsub_rn(1.f, acc), fmaf(c.y, inv_b, p.large_step_prob));
      c.radiance = add(c.radiance, scale(w_old, c.L));
      const float w_new = __fdiv_rn(__fadd_rn(acc, m.large_step ? 1.f : 0.f), fmaf(yn, inv_b, p.large_step_prob));
      if (lcg_next(c.cs) < acc) {
        ++accepted;
        splat(p.film, c.pix, scale(p.inv_eff_spp, c.radiance));
        c.radiance = scale(w_new, Ln);
        c.pix = c.npix;
        c.L = Ln;
        c.y = yn;
        m.accept();
      } else {
        if (acc > 0.f) splat(p.film, c.npix, scale(__fmul_rn(w_new, p.inv_eff_spp), Ln));
        m.reject();
      }
    }
    if (++c.it >= p.mutations_per_chain) {
      splat(p.film, c.pix, scale(p.inv_eff_spp, c.radiance));
      c.chain = -1;
    }
    put(c);
  }

  // the next mutation of the lane's chain, or the starting path of the next chain
  __device__ __forceinline__ bool start(Ray* ray, MltSampler* m) {
    ChainState c = get();
    if (c.chain < 0) {
      const unsigned long long i = claim_next(p.next);
      if (i >= static_cast<unsigned long long>(p.n_chains)) return false;
      c.chain = static_cast<int>(i);
      IndepSampler cs{xxhash32_two(static_cast<uint32_t>(p.frame_id), static_cast<uint32_t>(c.chain))};
      // AliasTable.Sample over the bootstrap weights (Util/AliasTable.fs:52-62)
      const float u = __fmul_rn(cs.next(), static_cast<float>(p.n_bootstrap));
      c.bid = min(static_cast<int>(u), p.n_bootstrap - 1);
      if (p.alias_prob) {
        const float frac = __fsub_rn(u, static_cast<float>(c.bid));
        if (frac >= p.alias_prob[c.bid]) c.bid = p.alias_idx[c.bid];
      }
      c.cs = cs.state;
      c.radiance = c.L = mk(0.f, 0.f, 0.f);
      c.y = 0.f;
      c.pix = 0;
      c.it = -1;
      m->inner = xxhash32_two(static_cast<uint32_t>(p.frame_id), static_cast<uint32_t>(c.bid));
      m->large_step = false;
      m->last_large = 0;
      m->cur_iter = 0;
      m->index = 0;
      m->initialized = 0;
      m->fresh = 0;
      m->X = p.X + static_cast<long long>(c.chain) * p.n_dims;
    }
    m->start_iteration();
    const DevView& v = *p.view;
    int nx, ny;
    *ray = mlt_camera(v, *m, &nx, &ny);
    c.npix = (v.height - ny - 1) * v.width + nx;
    put(c);
    return true;
  }
};

// 65,536 chains of a 512^2 render (Cornell with objects, Kelemen) took 94.5 ms as a plain loop per
// chain in lockstep (4.1 lanes active, 205 KB of code, no instruction to issue 12 cycles out of
// 16); on the path machine 91, with one copy of the draws (113 KB) 60, with the
// normalisations called 54.9; 4,096 chains 383 -> 203 ms.  4 blocks per SM (128 registers, no spills since
// the walk's state is small enough) against 3 (141), both with service at an eighth: 65,536 chains 53.0 and 52.7
// ms, 262,144 chains 44.0 and 45.3, 4,096 chains 193 and 200; in the Cornell box 34.5 and 35.9; with the
// Gaussian strategy 62.2 and 60.9, 262,144 chains 51.8 and 52.7.
constexpr int kChainBlocks = 4;

// kKelemen: the mutation strategy fixed at compile time (1 Kelemen, 0 Gaussian), so the kernel
// holds one strategy's code
template <bool kWT, int kWalk, int kKelemen>
__global__ void __launch_bounds__(kMachineThreads, kChainBlocks) k_mlt_chains(MltParams p, int lanes) {
  __shared__ float chain_block[kChainWords * kMachineThreads];
  MltTask task(p, chain_block);
  MltSampler m{};
  m.p_large = p.large_step_prob;
  m.kelemen = kKelemen;
  m.sigma = p.sigma;
  m.eps_min = p.eps_min;
  m.eps_max = p.eps_max;
  m.log_eps = logf(__fdiv_rn(m.eps_max, m.eps_min));
  m.stride = 1;
  m.max_dims = p.n_dims;
  path_machine<kWT, kWalk, false, true>(p.scene, task, m, p.max_depth, p.rr_depth, lanes);
  unsigned long long a = task.accepted;
  for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
  if ((threadIdx.x & 31) == 0 && a) atomicAdd(p.accepted, a);
}

template <class K>
cudaError_t launch(K kernel, const MltParams& p, long long n, cudaStream_t st) {
  const cudaError_t e = cudaMemsetAsync(p.next, 0, sizeof(*p.next), st);
  if (e != cudaSuccess) return e;
  const int grid = static_cast<int>(std::min<long long>(n, resident_grid(kernel, kMachineThreads)));
  kernel<<<grid, kMachineThreads, 0, st>>>(p, machine_lanes(n, static_cast<long long>(grid) * (kMachineThreads / 32)));
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_mlt_bootstrap(const MltParams& p, cudaStream_t st) {
  // while (depth < maxDepth) never runs: every luminance is zero
  if (p.max_depth <= 0) return cudaMemsetAsync(p.weights, 0, static_cast<size_t>(p.n_bootstrap) * sizeof(float), st);
  cudaError_t e = cudaSuccess;
  dispatch_walk<false>(p.scene, p.watertight, false, [&](auto wt, auto walk) {
    e = launch(k_mlt_bootstrap<decltype(wt)::value, decltype(walk)::value>, p, p.n_bootstrap, st);
  });
  return e;
}

cudaError_t launch_mlt_chains(const MltParams& p, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  dispatch_walk<false>(p.scene, p.watertight, false, [&](auto wt, auto walk) {
    constexpr bool kWT = decltype(wt)::value;
    constexpr int kWalk = decltype(walk)::value;
    e = p.kelemen ? launch(k_mlt_chains<kWT, kWalk, 1>, p, p.n_chains, st)
                  : launch(k_mlt_chains<kWT, kWalk, 0>, p, p.n_chains, st);
  });
  return e;
}

}  // namespace bn
