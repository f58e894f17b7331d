// bn_forward / bn_backward: differentiable material slots over the uploaded scene.
#include <cmath>
#include <string>
#include <vector>

#include "../device/adjoint.hpp"
#include "context.hpp"

namespace {

int prepare(bn_context* ctx, const bn_adjoint_desc* d, const float* params, const float* sparams, bn::AdjParams* p) {
  if (!ctx->has_scene) return ctx->fail(BN_ERR_NO_SCENE, "adjoint before bn_scene_upload");
  if (!d || !params) return ctx->fail(BN_ERR_INVALID_ARG, "adjoint: null descriptor or parameters");
  if (d->n_slots <= 0 || d->emissive_slot_base < 0 || d->emissive_slot_base > d->n_slots)
    return ctx->fail(BN_ERR_INVALID_ARG, "adjoint: bad slot counts");
  if (d->width <= 0 || d->height <= 0 || d->spp <= 0 || d->max_depth < 0 || d->rr_depth < 0)
    return ctx->fail(BN_ERR_INVALID_ARG, "adjoint: bad film, spp or depth");
  if (d->emissive_slot_base > ctx->scene.n_mats)
    return ctx->fail(BN_ERR_INVALID_ARG, "adjoint: material slots beyond the scene's materials");
  cudaError_t e;
  const size_t np = static_cast<size_t>(d->n_slots) * bn::kSlotParams;
  const long long pixels = static_cast<long long>(d->width) * d->height;
  if ((e = ctx->reserve(ctx->adj_params, 2 * np * sizeof(float))) != cudaSuccess) return ctx->cuda_fail(e, "adjoint params");
  if ((e = ctx->reserve(ctx->adj_aux, static_cast<size_t>(pixels) * d->spp * sizeof(float4))) != cudaSuccess)
    return ctx->cuda_fail(e, "adjoint path radiance");
  if ((e = ctx->reserve(ctx->adj_image, static_cast<size_t>(pixels) * 3 * sizeof(float))) != cudaSuccess)
    return ctx->cuda_fail(e, "adjoint image");
  if ((e = ctx->reserve(ctx->views, sizeof(bn::DevView))) != cudaSuccess) return ctx->cuda_fail(e, "adjoint view");
  bn_view v{};
  v.camera = d->camera;
  v.width = d->width;
  v.height = d->height;
  const bn::DevView dv = bnc::make_dev_view(v, 0, 0);
  float* dparams = ctx->adj_params.as<float>();
  float* dsparams = dparams + np;
  cudaStream_t st = ctx->stream;
  cudaMemcpyAsync(ctx->views.ptr, &dv, sizeof(dv), cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(dparams, params, np * sizeof(float), cudaMemcpyHostToDevice, st);
  const float* sp = (d->freeze_sampling && sparams) ? sparams : params;
  cudaMemcpyAsync(dsparams, sp, np * sizeof(float), cudaMemcpyHostToDevice, st);
  *p = bn::AdjParams{};
  p->scene = ctx->scene;
  p->view = ctx->views.as<bn::DevView>();
  p->n_slots = d->n_slots;
  p->emissive_base = d->emissive_slot_base;
  p->spp = d->spp;
  p->max_depth = d->max_depth;
  p->rr_depth = d->rr_depth;
  p->frame_id = d->frame_id;
  p->params = dparams;
  p->sparams = dsparams;
  p->path_L = ctx->adj_aux.as<float4>();
  p->image = ctx->adj_image.as<float>();
  p->n_pixels = pixels;
  return BN_OK;
}

// Whether the paths are those of an ordinary render of a patched scene (k_adjoint.cu): sampling
// follows the values, and no value makes a product of the patched form 0 or NaN where the two-material
// form's is not (a light's scale of 0 still has a derivative; non-finite parameters).
bool follows(const bn_adjoint_desc* d, const float* params, const float* sparams) {
  if ((d->freeze_sampling && sparams) || d->max_depth <= 0) return false;
  if (static_cast<long long>(d->width) * d->height > 0x7fffffffLL / d->spp) return false;
  for (int k = 0; k < d->n_slots * bn::kSlotParams; ++k)
    if (!std::isfinite(params[k])) return false;
  for (int k = d->emissive_slot_base; k < d->n_slots; ++k)
    if (!(params[bn::kSlotParams * k + 5] > 1e-20f)) return false;
  return true;
}

// device memory for the patched scene, and with `record` for the vertices; false: not to be had
bool patch_buffers(bn_context* ctx, const bn_adjoint_desc* d, bn::AdjParams* p, bool record) {
  const long long n = p->n_pixels * d->spp;
  const size_t mats = static_cast<size_t>(ctx->scene.n_mats + 1) * sizeof(bn::DevMaterial);
  const size_t lights = static_cast<size_t>(ctx->n_lights + 1) * sizeof(bn::DevLight);
  cudaError_t e = ctx->reserve(ctx->adj_scene, mats + lights);
  p->patched = ctx->scene;
  if (e == cudaSuccess && record) {
    // 17 bytes a vertex, up to 4 GB of them; longer paths are traced again in the adjoint
    if (n > (4LL << 30) / 17 / d->max_depth) return false;
    e = ctx->reserve(ctx->adj_rec, static_cast<size_t>(n) * d->max_depth * (sizeof(float4) + 1));
    p->rec = ctx->adj_rec.as<float4>();
    p->lit = reinterpret_cast<unsigned char*>(p->rec + n * d->max_depth);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  auto* m = ctx->adj_scene.as<bn::DevMaterial>();
  p->patched.mats = m;
  p->patched.lights = reinterpret_cast<bn::DevLight*>(m + ctx->scene.n_mats + 1);
  p->next = reinterpret_cast<unsigned long long*>(static_cast<char*>(ctx->error_word.ptr) + 64);
  return true;
}

// path_L of every path (and rec, lit), in the form that is faster at this many paths (the line is the
// megakernel renders', capi.cu); *ms is the device time before ctx->ev0, *launches the kernels
int follow_paths(bn_context* ctx, const bn_adjoint_desc* d, const bn::AdjParams& p, float* ms, int* launches) {
  const long long n = p.n_pixels * d->spp;
  cudaStream_t st = ctx->stream;
  cudaError_t e;
  cudaEventRecord(ctx->ev0, st);
  if (p.lit) cudaMemsetAsync(p.lit, 0, static_cast<size_t>(n) * d->max_depth, st);
  if ((e = bn::launch_adj_patch(p, const_cast<bn::DevMaterial*>(p.patched.mats), const_cast<bn::DevLight*>(p.patched.lights),
                                ctx->n_lights, st)) != cudaSuccess)
    return ctx->cuda_fail(e, "adjoint scene launch");
  bool ran = false;
  if (n >= bnc::kQueuePaths) {
    bn_render_desc r{};
    r.integrator = BN_INTEGRATOR_PATH;
    r.spp = d->spp;
    r.max_depth = d->max_depth;
    r.rr_depth = d->rr_depth;
    r.frame_id = d->frame_id;
    const int rc = bnc::wavefront_paths(ctx, p.patched, &r, n, {p.path_L, p.rec, p.lit}, &ran);
    if (rc) return rc;
    *ms = ctx->stats.last_kernel_ms;
    *launches = ctx->stats.last_launches + 1;
    cudaEventRecord(ctx->ev0, st);
  }
  if (!ran) {
    if ((e = bn::launch_adj_paths(p, st)) != cudaSuccess) return ctx->cuda_fail(e, "adjoint paths launch");
    *launches = 2;
  }
  return BN_OK;
}

}  // namespace

extern "C" int bn_forward(bn_context* ctx, const bn_adjoint_desc* d, const float* params, const float* sampling_params,
                          float* out_image) {
  if (!ctx) return BN_ERR_INVALID_ARG;
  cudaSetDevice(ctx->device);
  bn::AdjParams p;
  int rc = prepare(ctx, d, params, sampling_params, &p);
  if (rc) return rc;
  cudaError_t e;
  float ms_paths = 0.f;
  int launches = 0;
  // about one path per lane of the machine: the plain kernel's warps of 32 neighbours are as good
  // (36,864 / 51,200 / 102,400 / 163,840 / 240,000 paths 0.84 0.86 1.12 1.16 1.36 ms against 0.80 0.90 1.20 1.20 1.28)
  const long long n = p.n_pixels * d->spp;
  const bool one_round = n >= 49152 && n < 196608;
  if (!one_round && follows(d, params, sampling_params) && patch_buffers(ctx, d, &p, false)) {
    if ((rc = follow_paths(ctx, d, p, &ms_paths, &launches)) != BN_OK) return rc;
  } else {
    cudaEventRecord(ctx->ev0, ctx->stream);
    launches = 1;
    if ((e = bn::launch_adj_forward(p, ctx->stream)) != cudaSuccess) return ctx->cuda_fail(e, "forward launch");
  }
  cudaEventRecord(ctx->ev1, ctx->stream);
  if ((e = bn::launch_adj_image(p, ctx->stream)) != cudaSuccess) return ctx->cuda_fail(e, "image launch");
  cudaEventRecord(ctx->ev2, ctx->stream);
  if (out_image)
    cudaMemcpyAsync(out_image, p.image, static_cast<size_t>(p.n_pixels) * 3 * sizeof(float), cudaMemcpyDeviceToHost,
                    ctx->stream);
  if ((e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess) return ctx->cuda_fail(e, "forward");
  float ms_main = 0.f, ms_all = 0.f;
  cudaEventElapsedTime(&ms_main, ctx->ev0, ctx->ev1);
  cudaEventElapsedTime(&ms_all, ctx->ev0, ctx->ev2);
  ctx->stats.last_dominant_ms = ms_paths + ms_main;
  ctx->stats.last_kernel_ms = ms_paths + ms_all;
  ctx->stats.last_launches = launches + 1;
  ctx->stats.paths += static_cast<uint64_t>(p.n_pixels) * p.spp;
  return bnc::check_device_error(ctx);
}

extern "C" int bn_backward(bn_context* ctx, const bn_adjoint_desc* d, const float* params, const float* sampling_params,
                           const float* target_image, double* d_params, double* loss) {
  if (!ctx) return BN_ERR_INVALID_ARG;
  if (!target_image || !d_params) return ctx->fail(BN_ERR_INVALID_ARG, "bn_backward: null target or gradient");
  cudaSetDevice(ctx->device);
  bn::AdjParams p;
  int rc = prepare(ctx, d, params, sampling_params, &p);
  if (rc) return rc;
  cudaError_t e;
  const size_t np = static_cast<size_t>(d->n_slots) * bn::kSlotParams;
  if ((e = ctx->reserve(ctx->adj_target, static_cast<size_t>(p.n_pixels) * 3 * sizeof(float))) != cudaSuccess)
    return ctx->cuda_fail(e, "adjoint target");
  if ((e = ctx->reserve(ctx->adj_grad, (np + 1) * sizeof(double))) != cudaSuccess) return ctx->cuda_fail(e, "adjoint gradient");
  cudaStream_t st = ctx->stream;
  cudaMemcpyAsync(ctx->adj_target.ptr, target_image, static_cast<size_t>(p.n_pixels) * 3 * sizeof(float),
                  cudaMemcpyHostToDevice, st);
  cudaMemsetAsync(ctx->adj_grad.ptr, 0, (np + 1) * sizeof(double), st);
  p.target = ctx->adj_target.as<float>();
  p.grad = ctx->adj_grad.as<double>();
  p.loss = p.grad + np;
  float ms_paths = 0.f;
  int launches = 0;
  const bool replay = follows(d, params, sampling_params) && patch_buffers(ctx, d, &p, true);
  if (replay) {
    if ((rc = follow_paths(ctx, d, p, &ms_paths, &launches)) != BN_OK) return rc;
  } else {
    cudaEventRecord(ctx->ev0, st);
    launches = 1;
    if ((e = bn::launch_adj_forward(p, st)) != cudaSuccess) return ctx->cuda_fail(e, "adjoint forward launch");
  }
  if ((e = bn::launch_adj_image(p, st)) != cudaSuccess) return ctx->cuda_fail(e, "adjoint image launch");
  if ((e = bn::launch_adj_loss(p, st)) != cudaSuccess) return ctx->cuda_fail(e, "loss launch");
  cudaEventRecord(ctx->ev1, st);
  if ((e = replay ? bn::launch_adj_replay(p, st) : bn::launch_adj_backward(p, st)) != cudaSuccess) return ctx->cuda_fail(e, "backward launch");
  cudaEventRecord(ctx->ev2, st);
  std::vector<double> host(np + 1);
  cudaMemcpyAsync(host.data(), ctx->adj_grad.ptr, (np + 1) * sizeof(double), cudaMemcpyDeviceToHost, st);
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return ctx->cuda_fail(e, "backward");
  for (size_t i = 0; i < np; ++i) d_params[i] = host[i];
  if (loss) *loss = host[np];
  float ms_replay = 0.f, ms_all = 0.f;
  cudaEventElapsedTime(&ms_replay, ctx->ev1, ctx->ev2);
  cudaEventElapsedTime(&ms_all, ctx->ev0, ctx->ev2);
  ctx->stats.last_dominant_ms = ms_replay;
  ctx->stats.last_kernel_ms = ms_paths + ms_all;
  ctx->stats.last_launches = launches + 3;
  return bnc::check_device_error(ctx);
}
