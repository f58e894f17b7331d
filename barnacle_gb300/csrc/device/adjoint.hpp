// Differentiable-material render (forward) and path-replay adjoint (backward) parameters.
#pragma once
#include <cuda_runtime.h>

#include "dev_types.cuh"

namespace bn {

constexpr int kSlotParams = 6;  // albedo r, g, b, roughness, metallic, emission scale

struct AdjParams {
  DevScene scene;
  const DevView* view;
  int n_slots, emissive_base;
  int spp, max_depth, rr_depth, frame_id;
  const float* params;        // values: n_slots * 6
  const float* sparams;       // sampling decisions: n_slots * 6 (== params unless frozen)
  float4* path_L;             // radiance of path pixel * spp + sample
  // a run whose sampling follows the values it renders (sparams == params): the scene with the
  // slots' materials and the scaled lights, and for the adjoint the paths' vertices (WfParams::rec)
  DevScene patched;
  float4* rec;
  unsigned char* lit;
  unsigned long long* next;   // the next path a lane of the path machine claims
  float* image;               // W*H*3, Film.Pixels order
  const float* target;        // W*H*3
  double* grad;               // n_slots * 6
  double* loss;               // 1
  long long n_pixels;
};

// p.patched's materials and lights (n_lights) from p.scene's and p.params
cudaError_t launch_adj_patch(const AdjParams& p, DevMaterial* mats, DevLight* lights, int n_lights, cudaStream_t st);
// the paths of p.patched on the path machine: path_L, and rec and lit if p.rec is set
cudaError_t launch_adj_paths(const AdjParams& p, cudaStream_t st);
// the adjoint from path_L, rec and lit
cudaError_t launch_adj_replay(const AdjParams& p, cudaStream_t st);
cudaError_t launch_adj_forward(const AdjParams& p, cudaStream_t st);
cudaError_t launch_adj_image(const AdjParams& p, cudaStream_t st);
cudaError_t launch_adj_loss(const AdjParams& p, cudaStream_t st);
cudaError_t launch_adj_backward(const AdjParams& p, cudaStream_t st);

}  // namespace bn
