// bn_context: the device-resident state behind the C-ABI.
#pragma once
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "../../../include/barnacle_gpu.h"
#include "../device/dev_types.cuh"
#include "../device/launch.hpp"
#include "../device/pssmlt.hpp"
#include "dev_buf.hpp"

namespace bnc {
constexpr size_t kPinnedBytes = 65536;
// the GPU BVH builder's buffers (bvh_gpu.cu)
struct BvhWork {
  DevBuf bounds, items, ranges, level, nodes, out, perm, odd, counters;
  DevBuf vertices, indices, slots, scene_odd, wide;  // bn_scene_upload's meshes
  void* host_counters = nullptr;  // pinned
  void trim();                    // frees what is too large to keep
  void release();
};
// trims a call's buffers however the call ends
struct TrimAtExit {
  BvhWork& work;
  ~TrimAtExit() { work.trim(); }
};
}  // namespace bnc

struct bn_context {
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev2 = nullptr;
  std::string err;
  char* pinned = nullptr;  // bnc::kPinnedBytes of pinned host memory: the error word, then short results

  // scene
  bool has_scene = false;
  bn::DevScene scene{};
  // error_word: 256 bytes, the BN_DEVERR_* word at 0, the counter of claimed items at 64
  DevBuf nodes, nodes4, tris, inst, mats, lights, light_inst, tri_pdf, tri_lights, error_word, counters;
  std::vector<int32_t> inst_order;     // TLAS order -> descriptor index
  std::vector<bn::DevMaterial> host_mats;
  std::vector<int32_t> host_inst_light;  // per TLAS instance: light index
  int n_lights = 0;
  float scene_lo[3] = {0.f, 0.f, 0.f}, scene_hi[3] = {0.f, 0.f, 0.f};  // TLAS root box
  bool scene_simple = false;  // Lambertian materials, triangle meshes, the uniform light sampler
  // failure-detection limits (bn_set_limits; 0 = the defaults)
  int limit_stack = 0;        // traversal stack entries a walk may use
  int limit_iters = 0;        // wavefront bounce-loop iterations before the watchdog stops it

  // queries
  DevBuf q_in, q_out;

  // render
  DevBuf views, item_offsets, partial, film, wf_state, rgba;
  long long film_floats = 0;
  bn_stats stats{};

  bnc::BvhWork bvh;

  // pssmlt / adjoint scratch
  DevBuf mlt_state, mlt_boot, mlt_chain, adj_params, adj_image, adj_target, adj_grad, adj_aux, adj_scene, adj_rec;

  // wavefront path state, captured graph and launch shape (owned by wavefront.cu)
  void* wf = nullptr;
  void (*wf_release)(void*) = nullptr;
  bool (*wf_spare)(void*) = nullptr;  // gives the path state back; false: there was none
  long long scene_generation = 0;  // bumped by every bn_scene_upload

  // Room in one of the context's buffers.  The wavefront's path state, which stays with the context from
  // render to render (18 GB after one of 64 M paths), goes when the GPU has no other memory left.
  // (Allocating it per call instead took 1.6 of 6.5 ms of a Cornell render, 12 of 211 of 16 instanced views.)
  cudaError_t reserve(DevBuf& b, size_t n) {
    cudaError_t e = b.reserve(n);
    if (e == cudaErrorMemoryAllocation && wf_spare && wf_spare(wf)) e = b.reserve(n);
    return e;
  }
  int fail(int code, const std::string& msg) {
    err = msg;
    return code;
  }
  int cuda_fail(cudaError_t e, const char* where) {
    err = std::string(where) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? BN_ERR_OUT_OF_MEMORY : BN_ERR_CUDA;
  }
};

namespace bnc {
// host-side view constants (Extensions/Camera/Pinhole.fs:16-22), shared by all render modes
bn::DevView make_dev_view(const bn_view& v, long long pixel_offset, long long path_offset);
// Waits for the stream and reports the device error word (BN_ERR_DEVICE, the word cleared); or the
// same in two parts around a wait that the call makes anyway.
int check_device_error(bn_context* ctx);
void queue_device_error(bn_context* ctx);
int queued_device_error(bn_context* ctx);
// The plain megakernel's sample chunks: each work item runs spc consecutive samples of one pixel,
// chunks = ceil(spp / spc) items per pixel.  max_items > 0 caps pixels * chunks (fixed scratch).
struct MegaChunks {
  int chunks = 1, spc = 1;
};
MegaChunks mega_chunks(long long pixels, int spp, long long max_items);
// Launch parameters of the megakernel shared by bn_render and bn_render_noalloc (views, item
// offsets, partial sums, film and counting are filled in by the caller).
bn::MegaParams mega_params(const bn_context* ctx, const bn_render_desc* d, const std::vector<bn::DevView>& views,
                           const MegaChunks& ck, long long items, long long pixels);
// Paths from which on a render's paths run in the wavefront's queues, whose sorted rays keep 15 to 26 of
// a warp's 32 lanes walking where the path machine's lanes keep 9 to 11.  Kernel ms on the machine / in
// the queues: Cornell box at 393,216 and 786,432 paths 1.03 / 0.95 and 1.95 / 1.40 (196,608: 0.56 / 0.77),
// Cornell with objects at 524,288 and 786,432 3.23 / 4.04 and 4.72 / 4.65, material forward 2.07 / 2.45 and 2.97 /
// 2.74, material gradient 2.62 / 2.92 and 3.74 / 3.46, an instanced view at 2 and 3 spp 10.76 / 10.74 and 13.5 / 13.6.
constexpr long long kQueuePaths = 3 << 18;
// A megakernel-mode render (p: its launch parameters) whose paths run in the wavefront's queues and
// are summed in the mode's order.  *ran stays false, with nothing rendered, when the path state
// does not fit the GPU's free memory.
int render_ordered(bn_context* ctx, const bn_render_desc* d, const bn::MegaParams& p, bool* ran);
// Where an ordered run of the wavefront leaves its paths (WfParams::path_L, rec, lit).
struct PathRecords {
  float4* L;
  float4* rec;
  unsigned char* lit;
};
// The n_paths camera paths of the one view in ctx->views through the wavefront's queues.  *ran stays
// false when the path state does not fit the GPU's free memory.
int wavefront_paths(bn_context* ctx, const bn::DevScene& scene, const bn_render_desc* d, long long n_paths,
                    const PathRecords& out, bool* ran);
// bn_set_memory_limit: bytes of path state that a call may ask for (0: what the GPU has)
void set_path_memory_limit(bn_context* ctx, size_t bytes);
int render_wavefront(bn_context* ctx, const bn_render_desc* d, const std::vector<bn::DevView>& views);
// BVHNode.Build on the GPU (bvh_gpu.cu): the host builder's nodes and permutation
int gpu_bvh_build(bn_context* ctx, const float* bounds, int32_t n, std::vector<bn_bvh_node>* nodes,
                  std::vector<int32_t>* perm);
// the same from n > 0 boxes in device memory, left there: ctx->bvh.out, perm, and with `odd` the
// parity of each node's depth in ctx->bvh.odd.  *nan: not built, a box is for the host builder.
int gpu_bvh_build_resident(bn_context* ctx, const float* bounds_device, int32_t n, bool odd, bool* nan, int* n_nodes);
int render_pssmlt(bn_context* ctx, const bn_render_desc* d, const std::vector<bn::DevView>& views);
// the PSSMLT chains in the wavefront (wavefront.cu), after the bootstrap
int render_pssmlt_wavefront(bn_context* ctx, const bn_render_desc* d, const bn::MltParams& mp, int* launches);
}  // namespace bnc
