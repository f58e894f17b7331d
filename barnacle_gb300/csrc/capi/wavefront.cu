// Wavefront render orchestration: path-state buffers, the CUDA graph whose while-node runs the
// whole bounce loop on the device, the host-driven fallback loop, and the rule for the pool's size.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../device/pssmlt.hpp"
#include "../device/wavefront.hpp"
#include "context.hpp"
#include "path_state.hpp"

namespace {

struct WfState {
  bnc::PathState paths;
  DevBuf params, counters, work_next, hist, off;  // of one size, whatever the pool
  DevBuf film_acc;
  DevBuf mlt_smp, mlt_chain;  // PSSMLT chains: sampler state and chain records
  // captured graph (one per launch shape)
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaGraphConditionalHandle cond = 0;
  bool graph_failed = false;
  bn::WfLaunch shape{};
  int shape_cap = -1;
  // the PSSMLT iteration's second stream and its fork / join events (made on first use)
  bn::WfFork fork{nullptr, nullptr, nullptr};

  cudaError_t ensure_fork() {
    cudaError_t e = cudaSuccess;
    if (!fork.side) e = cudaStreamCreateWithFlags(&fork.side, cudaStreamNonBlocking);
    if (e == cudaSuccess && !fork.fork) e = cudaEventCreateWithFlags(&fork.fork, cudaEventDisableTiming);
    if (e == cudaSuccess && !fork.join) e = cudaEventCreateWithFlags(&fork.join, cudaEventDisableTiming);
    return e;
  }

  void release() {
    paths.release();
    for (DevBuf* x : {&params, &counters, &work_next, &hist, &off, &film_acc, &mlt_smp, &mlt_chain}) x->release();
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    exec = nullptr;
    graph = nullptr;
    if (fork.fork) cudaEventDestroy(fork.fork);
    if (fork.join) cudaEventDestroy(fork.join);
    if (fork.side) cudaStreamDestroy(fork.side);
    fork = bn::WfFork{nullptr, nullptr, nullptr};
  }
};

WfState* state(bn_context* ctx) {
  if (!ctx->wf) {
    ctx->wf = new WfState();
    ctx->wf_release = [](void* p) {
      auto* s = static_cast<WfState*>(p);
      s->release();
      delete s;
    };
    ctx->wf_spare = [](void* p) {
      auto* s = static_cast<WfState*>(p);
      const bool held = s->paths.held() > 0;
      s->paths.release();
      return held;
    };
  }
  return static_cast<WfState*>(ctx->wf);
}

// what a run of `pool` slots works in, and `paths` radiances of an ordered one
cudaError_t ensure_pool(WfState* w, int pool, long long paths = 0) {
  cudaError_t e = w->paths.reserve(static_cast<size_t>(pool), static_cast<size_t>(paths));
  if (e == cudaSuccess) e = w->params.reserve(sizeof(bn::WfParams));
  if (e == cudaSuccess) e = w->counters.reserve(bn::kCntSize * sizeof(int));
  if (e == cudaSuccess) e = w->work_next.reserve(sizeof(unsigned long long));
  if (e == cudaSuccess) e = w->hist.reserve(2 * bn::kSortBins * sizeof(unsigned));
  if (e == cudaSuccess) e = w->off.reserve((bn::kSortBins + bn::kSortBins / 1024) * sizeof(unsigned));
  if (e != cudaSuccess) w->paths.release();
  return e;
}

// Path slots of a render that does not choose them: one per path, up to 64 M (16 GB).  Every path
// then starts at once, the queues are as long and the sorted rays as coherent as they can be, and
// a bounce is one iteration; fewer slots cost more, short iterations, more slots only add rows to
// scan.  Measured (kernel ms by log2 of the slots, the render's paths in brackets): Cornell box
// [2^22] 20: 6.07, 21: 5.43, 22: 4.90, 23: 5.00; Cornell with objects [2^23] 21: 20.8, 22: 18.5,
// 23: 17.0, 24: 17.0; 16 instanced views [2^25.8] 22: 230.5, 23: 218.2, 24: 211.1, 25: 205.5, 26: 199.5.
// A cap of 2 blocks per SM was 1.8 times slower at every one of them.
int default_pool(long long paths) {
  return static_cast<int>(std::min<long long>(1LL << 26, (paths + 1023) / 1024 * 1024));
}

// the while-node graph of the path tracer: body = one iteration (regen, extend, shade, shadow,
// control)
int build_graph(bn_context* ctx, WfState* w) {
  if (w->exec) {
    cudaGraphExecDestroy(w->exec);
    w->exec = nullptr;
  }
  if (w->graph) {
    cudaGraphDestroy(w->graph);
    w->graph = nullptr;
  }
  cudaError_t e;
  if ((e = cudaGraphCreate(&w->graph, 0)) != cudaSuccess) return ctx->cuda_fail(e, "cudaGraphCreate");
  if ((e = cudaGraphConditionalHandleCreate(&w->cond, w->graph, 1, cudaGraphCondAssignDefault)) != cudaSuccess)
    return ctx->cuda_fail(e, "cudaGraphConditionalHandleCreate");
  cudaGraphNodeParams np{};
  np.type = cudaGraphNodeTypeConditional;
  np.conditional.handle = w->cond;
  np.conditional.type = cudaGraphCondTypeWhile;
  np.conditional.size = 1;
  cudaGraphNode_t node;
  if ((e = cudaGraphAddNode(&node, w->graph, nullptr, nullptr, 0, &np)) != cudaSuccess)
    return ctx->cuda_fail(e, "cudaGraphAddNode(while)");
  cudaGraph_t body = np.conditional.phGraph_out[0];
  if ((e = cudaStreamBeginCaptureToGraph(ctx->stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed)) !=
      cudaSuccess)
    return ctx->cuda_fail(e, "cudaStreamBeginCaptureToGraph");
  cudaError_t le = bn::wf_launch_iteration(w->params.as<bn::WfParams>(), w->shape, true, ctx->stream);
  cudaGraph_t captured = body;
  e = cudaStreamEndCapture(ctx->stream, &captured);
  if (le != cudaSuccess) return ctx->cuda_fail(le, "capture of the bounce loop");
  if (e != cudaSuccess) return ctx->cuda_fail(e, "cudaStreamEndCapture");
  if ((e = cudaGraphInstantiate(&w->exec, w->graph, 0)) != cudaSuccess) return ctx->cuda_fail(e, "cudaGraphInstantiate");
  return BN_OK;
}

// The bounce loop over path ids [first, end): into w->film_acc and ctx->film, or with `ordered` into
// its buffers.
int run(bn_context* ctx, WfState* w, const bn::DevScene& scene, const bn_render_desc* d, long long n_pixels,
        long long first, long long end, int n_views, int pool, int cap, bool use_graph, const bnc::PathRecords* ordered) {
  cudaError_t e;
  if ((e = ensure_pool(w, pool)) != cudaSuccess) return ctx->cuda_fail(e, "wavefront path-state allocation");
  if (!ordered && (e = w->film_acc.reserve(static_cast<size_t>(n_pixels) * 3 * sizeof(double))) != cudaSuccess)
    return ctx->cuda_fail(e, "wavefront film allocation");
  const bool wt = d->flags & BN_RENDER_WATERTIGHT;
  const bool wide = scene.wide != 0;
  // The ray queue is sorted by ray key: without it 8 to 10 % more.  Shadow rays are sorted in scenes of
  // many instances.  They are written in the order in which the sorted extension rays ended, and in a
  // scene of few instances that is order enough: kernel ms sorted / not, 16 instanced views of 4 spp (1,089
  // instances) 225.9 / 229.7, one view 16.92 / 16.95; Cornell box at 64 and 256 spp (8 instances) 5.44 / 5.28
  // and 20.4 / 19.6, Cornell with objects at 8, 32 and 128 spp (11) 7.45 / 7.31, 18.45 / 18.22 and 62.3 /
  // 61.4, materials at 32, 128 and 512 spp (14) 4.54 / 4.47, 12.15 / 12.18 and 43.1 / 43.6.  The line lies
  // between the measured 14 and 1,089.
  const bool sort = true, sort_shadow = scene.n_inst >= 128;
  const bool count = d->flags & BN_RENDER_COUNT;
  const int key_bits = bn::sort_key_bits(pool);
  if (w->shape_cap != cap || w->shape.watertight != wt || w->shape.wide != wide || w->shape.sort != sort ||
      w->shape.sort_shadow != sort_shadow || w->shape.count != count || w->shape.mlt ||
      w->shape.sort_tiles != (1 << (2 * key_bits + 6)) / 1024) {
    w->shape = bn::wf_launch_shape(wt, wide, sort, sort_shadow, count, cap, false, false, 0, key_bits);
    w->shape_cap = cap;
    if (w->exec) {
      cudaGraphExecDestroy(w->exec);
      w->exec = nullptr;
    }
  }
  const bn::DevScene walk = bn::walk_scene(scene);
  if (std::memcmp(&w->shape.walk, &walk, sizeof(walk)) != 0) {  // part of the captured launches
    w->shape.walk = walk;
    if (w->exec) {
      cudaGraphExecDestroy(w->exec);
      w->exec = nullptr;
    }
  }
  bn::WfParams p{};
  p.scene = scene;
  p.views = ctx->views.as<bn::DevView>();
  p.n_views = n_views;
  p.spp = d->spp;
  p.max_depth = d->max_depth;
  p.rr_depth = d->rr_depth;
  p.frame_id = d->frame_id;
  p.integrator = d->integrator;
  p.pool = pool;
  p.first_path = first;
  p.total_paths = end;
  p.n_pixels = n_pixels;
  p.max_iters = static_cast<int>(std::min<long long>(1LL << 30, ((end - first) / pool + 2) * (d->max_depth + 2) + 64));
  // bn_set_limits' cap is the wavefront mode's
  if (ctx->limit_iters > 0 && !ordered) p.max_iters = ctx->limit_iters;
  p.slot = w->paths.slot.as<float4>();
  p.q_active = w->paths.q_active.as<int>();
  p.q_done = w->paths.q_done.as<int>();
  p.sort = sort ? 1 : 0;
  p.sort_shadow = sort_shadow ? 1 : 0;
  {
    float lo[3], sc[3];
    for (int a = 0; a < 3; ++a) {
      const float ext = ctx->scene_hi[a] - ctx->scene_lo[a];
      lo[a] = ctx->scene_lo[a];
      sc[a] = ext > 0.f && std::isfinite(ext) ? (a == 1 ? 8.f : static_cast<float>(1 << key_bits)) / ext : 0.f;
    }
    p.key_lo = make_float4(lo[0], lo[1], lo[2], 0.f);
    p.key_scale = make_float4(sc[0], sc[1], sc[2], 0.f);
    p.key_bits = key_bits;
  }
  p.q_key = w->paths.q_key.as<int>();
  p.q_ray = sort ? w->paths.q_ray.as<int>() : w->paths.q_active.as<int>();
  p.sh_key = w->paths.sh_key.as<int>();
  p.q_shadow = w->paths.q_shadow.as<int>();
  p.hist = w->hist.as<unsigned>();
  p.off = w->off.as<unsigned>();
  p.q_bins = w->paths.q_bins.as<int>();
  p.shadow = w->paths.shadow.as<float4>();
  p.counters = w->counters.as<int>();
  p.trace_counters = ctx->counters.ptr;
  p.work_next = w->work_next.as<unsigned long long>();
  p.film_acc = w->film_acc.as<double>();
  if (ordered) {
    p.path_L = ordered->L;
    p.rec = ordered->rec;
    p.lit = ordered->lit;
  }
  p.film_out = ctx->film.as<float>();
  if (use_graph && !w->exec && !w->graph_failed) {
    if (build_graph(ctx, w) != BN_OK) {
      w->graph_failed = true;  // fall back to the host-driven loop; the message stays in ctx->err
      use_graph = false;
    }
  }
  if (use_graph && !w->exec) use_graph = false;
  p.cond = w->cond;
  cudaStream_t st = ctx->stream;
  cudaMemcpyAsync(w->params.ptr, &p, sizeof(p), cudaMemcpyHostToDevice, st);
  cudaMemsetAsync(w->counters.ptr, 0, bn::kCntSize * sizeof(int), st);
  for (int k = 0; k < 2; ++k)  // the bins in use of both queues' counts
    cudaMemsetAsync(w->hist.as<unsigned>() + k * bn::kSortBins, 0, (sizeof(unsigned) << (2 * key_bits + 6)), st);
  cudaMemsetAsync(w->work_next.ptr, 0, sizeof(unsigned long long), st);
  if (!ordered) cudaMemsetAsync(w->film_acc.ptr, 0, static_cast<size_t>(n_pixels) * 3 * sizeof(double), st);
  cudaEventRecord(ctx->ev0, st);
  int launches = 0;
  if (p.max_depth <= 0 && p.integrator == BN_INTEGRATOR_PATH) {
    // PathTracing: while (depth < maxDepth) never runs, every path's radiance is zero
    // (Normal and Direct ignore maxDepth)
  } else if (use_graph) {
    if ((e = cudaGraphLaunch(w->exec, st)) != cudaSuccess) return ctx->cuda_fail(e, "cudaGraphLaunch");
  } else {
    for (int it = 0; it < p.max_iters + 1; ++it) {
      if ((e = bn::wf_launch_iteration(w->params.as<bn::WfParams>(), w->shape, false, st)) != cudaSuccess)
        return ctx->cuda_fail(e, "wavefront iteration launch");
      launches += 5 + (sort ? 3 : 0) + (sort_shadow ? 3 : 0);
      int again = 0;
      cudaMemcpyAsync(&again, w->counters.as<int>() + bn::kCntAgain, sizeof(int), cudaMemcpyDeviceToHost, st);
      if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return ctx->cuda_fail(e, "wavefront iteration");
      if (!again) break;
    }
  }
  cudaEventRecord(ctx->ev1, st);
  if (!ordered && (e = bn::wf_launch_resolve(w->params.as<bn::WfParams>(), st)) != cudaSuccess)
    return ctx->cuda_fail(e, "wavefront resolve");
  cudaEventRecord(ctx->ev2, st);
  if ((e = cudaEventSynchronize(ctx->ev2)) != cudaSuccess) return ctx->cuda_fail(e, "wavefront render");
  int counters[bn::kCntSize];
  cudaMemcpy(counters, w->counters.ptr, sizeof(counters), cudaMemcpyDeviceToHost);
  float ms_loop = 0.f, ms_all = 0.f;
  cudaEventElapsedTime(&ms_loop, ctx->ev0, ctx->ev1);
  cudaEventElapsedTime(&ms_all, ctx->ev0, ctx->ev2);
  if (use_graph) launches = (5 + (sort ? 3 : 0) + (sort_shadow ? 3 : 0)) * counters[bn::kCntIter];
  ctx->stats.last_kernel_ms = ms_all;
  ctx->stats.last_dominant_ms = ms_loop;
  ctx->stats.last_launches = launches + (ordered ? 0 : 1);
  return BN_OK;
}

// The bounce loop of PSSMLT chains (one slot per chain), enqueued on the context's stream after
// the bootstrap as host-driven iterations: a render of 65,536 chains runs about 2,100 short ones,
// and measured at 1024^2 they took 435-454 ms as launches from the host against 489-500 ms as the
// iterations of a conditional graph node.  Splats go straight into ctx->film.  Returns the
// iterations run through *iters.
int run_mlt(bn_context* ctx, WfState* w, const bn_render_desc* d, const bn::MltParams& mp, int* iters) {
  cudaError_t e;
  const int pool = mp.n_chains;
  if ((e = ensure_pool(w, pool)) != cudaSuccess) return ctx->cuda_fail(e, "wavefront chain-state allocation");
  if ((e = w->ensure_fork()) != cudaSuccess) return ctx->cuda_fail(e, "wavefront chain stream");
  if ((e = w->mlt_smp.reserve(static_cast<size_t>(pool) * sizeof(int4))) != cudaSuccess ||
      (e = w->mlt_chain.reserve(static_cast<size_t>(pool) * 3 * sizeof(float4))) != cudaSuccess)
    return ctx->cuda_fail(e, "wavefront chain records");
  const bool wt = d->flags & BN_RENDER_WATERTIGHT;
  const bool wide = ctx->scene.wide != 0;
  const bool kelemen = mp.kelemen != 0;
  // 65,536 chains are few rays per launch: the queues are traversed unsorted
  const bn::WfLaunch want = bn::wf_launch_shape(wt, wide, false, false, false, 0, true, kelemen, pool);
  if (!w->shape.mlt || w->shape.watertight != wt || w->shape.wide != wide || w->shape.mlt_kelemen != kelemen ||
      w->shape.grid_extend != want.grid_extend || w->shape.grid_shadow != want.grid_shadow) {
    w->shape = want;
    w->shape_cap = -1;
    if (w->exec) {
      cudaGraphExecDestroy(w->exec);
      w->exec = nullptr;
    }
  }
  w->shape.walk = bn::walk_scene(ctx->scene);
  bn::WfParams p{};
  p.scene = ctx->scene;
  p.views = mp.view;
  p.n_views = 1;
  p.spp = d->spp;
  p.max_depth = d->max_depth;
  p.rr_depth = d->rr_depth;
  p.frame_id = d->frame_id;
  p.integrator = BN_INTEGRATOR_PSSMLT;
  p.pool = pool;
  p.total_paths = 0;
  p.n_pixels = 0;
  // a mutation's path takes at most max_depth iterations (at least one), and one more when its
  // last shadow record is traced after it ends
  p.max_iters = static_cast<int>(std::min<long long>(
      1LL << 30, (static_cast<long long>(mp.mutations_per_chain) + 1) * (std::max(1, d->max_depth) + 1) + 64));
  if (ctx->limit_iters > 0) p.max_iters = ctx->limit_iters;
  p.slot = w->paths.slot.as<float4>();
  p.q_active = w->paths.q_active.as<int>();
  p.q_done = w->paths.q_done.as<int>();
  p.sort = 0;
  p.sort_shadow = 0;
  p.key_bits = 5;
  p.q_ray = w->paths.q_active.as<int>();
  p.q_bins = w->paths.q_bins.as<int>();
  p.shadow = w->paths.shadow.as<float4>();
  p.counters = w->counters.as<int>();
  p.trace_counters = ctx->counters.ptr;
  p.work_next = w->work_next.as<unsigned long long>();
  p.film_out = mp.film;
  p.mlt = 1;
  bn::MltWf& q = p.mlt_p;
  q.n_chains = mp.n_chains;
  q.n_bootstrap = mp.n_bootstrap;
  q.n_dims = mp.n_dims;
  q.mutations = mp.mutations_per_chain;
  q.kelemen = mp.kelemen;
  q.p_large = mp.large_step_prob;
  q.sigma = mp.sigma;
  q.eps_min = mp.eps_min;
  q.eps_max = mp.eps_max;
  q.b = mp.b;
  q.inv_eff_spp = mp.inv_eff_spp;
  q.alias_prob = mp.alias_prob;
  q.alias_idx = mp.alias_idx;
  q.smp = w->mlt_smp.as<int4>();
  q.chain = w->mlt_chain.as<float4>();
  q.X = mp.X;
  q.film = mp.film;
  q.accepted = mp.accepted;
  cudaStream_t st = ctx->stream;
  cudaMemcpyAsync(w->params.ptr, &p, sizeof(p), cudaMemcpyHostToDevice, st);
  cudaMemsetAsync(w->counters.ptr, 0, bn::kCntSize * sizeof(int), st);
  cudaMemsetAsync(w->paths.slot.ptr, 0, static_cast<size_t>(pool) * 8 * sizeof(float4), st);  // every chain unstarted
  // (checking the loop condition every 4 or 16 iterations instead of every one measured slower:
  // 499 and 510 against 450 ms)
  for (int it = 0; it < p.max_iters + 1; ++it) {
    if ((e = bn::wf_launch_iteration(w->params.as<bn::WfParams>(), w->shape, false, st, &w->fork)) != cudaSuccess)
      return ctx->cuda_fail(e, "wavefront chain iteration launch");
    int again = 0;
    cudaMemcpyAsync(&again, w->counters.as<int>() + bn::kCntAgain, sizeof(int), cudaMemcpyDeviceToHost, st);
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return ctx->cuda_fail(e, "wavefront chain iteration");
    if (!again) break;
  }
  int counters[bn::kCntSize];
  e = cudaMemcpyAsync(counters, w->counters.ptr, sizeof(counters), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return ctx->cuda_fail(e, "wavefront chains");
  *iters = counters[bn::kCntIter];
  return BN_OK;
}

}  // namespace

namespace bnc {

int render_pssmlt_wavefront(bn_context* ctx, const bn_render_desc* d, const bn::MltParams& mp, int* launches) {
  int iters = 0;
  const int rc = run_mlt(ctx, state(ctx), d, mp, &iters);
  *launches = 5 * iters;
  return rc;
}

void set_path_memory_limit(bn_context* ctx, size_t bytes) {
  PathState& paths = state(ctx)->paths;
  paths.limit = bytes;
  if (bytes && paths.held() > bytes) paths.release();
}

int render_ordered(bn_context* ctx, const bn_render_desc* d, const bn::MegaParams& p, bool* ran) {
  // batches of whole pixels with at most 128 M paths (2 GB of radiances; half a second of work)
  const long long per = std::min<long long>(p.n_pixels, std::max<long long>(1, (1LL << 27) / d->spp));
  WfState* w = state(ctx);
  const int pool = std::max(default_pool(per * d->spp), 1024);
  cudaError_t e = ensure_pool(w, pool, per * d->spp);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    return BN_OK;  // *ran is false: the caller renders without path state
  }
  if (e != cudaSuccess) return ctx->cuda_fail(e, "wavefront path-state allocation");
  *ran = true;
  float loop_ms = 0.f, sum_ms = 0.f;
  int launches = 0;
  for (long long first = 0; first < p.n_pixels; first += per) {
    const long long n = std::min(per, p.n_pixels - first);
    const PathRecords out{w->paths.path_L.as<float4>(), nullptr, nullptr};
    const int rc = run(ctx, w, ctx->scene, d, p.n_pixels, first * d->spp, (first + n) * d->spp, p.n_views, pool, 0, true,
                       &out);
    if (rc) return rc;
    loop_ms += ctx->stats.last_dominant_ms;
    launches += ctx->stats.last_launches + 1;
    cudaEventRecord(ctx->ev0, ctx->stream);
    if ((e = bn::launch_mega_chunks(p, w->paths.path_L.as<float4>(), first, n, ctx->stream)) != cudaSuccess)
      return ctx->cuda_fail(e, "ordered sums");
    if (first + n == p.n_pixels) {
      ++launches;
      if ((e = bn::launch_mega_reduce(p, ctx->stream)) != cudaSuccess) return ctx->cuda_fail(e, "reduce launch");
    }
    cudaEventRecord(ctx->ev2, ctx->stream);
    if ((e = cudaEventSynchronize(ctx->ev2)) != cudaSuccess) return ctx->cuda_fail(e, "ordered sums");
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev2);
    sum_ms += ms;
  }
  ctx->stats.last_dominant_ms = loop_ms;
  ctx->stats.last_kernel_ms = loop_ms + sum_ms;
  ctx->stats.last_launches = launches;
  ctx->stats.paths += static_cast<uint64_t>(p.n_paths);
  return BN_OK;
}

int wavefront_paths(bn_context* ctx, const bn::DevScene& scene, const bn_render_desc* d, long long n_paths,
                    const PathRecords& out, bool* ran) {
  WfState* w = state(ctx);
  const int pool = std::max(default_pool(n_paths), 1024);
  const cudaError_t e = ensure_pool(w, pool);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    return BN_OK;
  }
  if (e != cudaSuccess) return ctx->cuda_fail(e, "wavefront path-state allocation");
  *ran = true;
  return run(ctx, w, scene, d, n_paths / d->spp, 0, n_paths, 1, pool, 0, true, &out);
}

int render_wavefront(bn_context* ctx, const bn_render_desc* d, const std::vector<bn::DevView>& views) {
  WfState* w = state(ctx);
  long long pixels = 0, total = 0;
  for (const auto& v : views) {
    pixels += static_cast<long long>(v.width) * v.height;
    total += static_cast<long long>(v.width) * v.height * d->spp;
  }
  const bool use_graph = !(d->flags & BN_RENDER_NO_GRAPH);
  const int cap = d->block_size;  // block_size doubles as the blocks/SM cap
  int pool = d->queue_capacity;
  if (pool <= 0) pool = default_pool(total);
  pool = std::max(pool, 1024);
  if (d->queue_capacity <= 0) {
    // a default pool gives way on a GPU whose memory others hold
    cudaError_t e;
    while ((e = ensure_pool(w, pool)) == cudaErrorMemoryAllocation && pool > (1 << 20)) {
      cudaGetLastError();
      pool >>= 1;
    }
  }
  const int rc = run(ctx, w, ctx->scene, d, pixels, 0, total, static_cast<int>(views.size()), pool, cap, use_graph, nullptr);
  if (rc) return rc;
  ctx->stats.paths += static_cast<uint64_t>(total);
  return BN_OK;
}

}  // namespace bnc
