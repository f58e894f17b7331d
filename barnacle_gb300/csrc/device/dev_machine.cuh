// The path machine: whole paths on persistent lanes.
//
// A loop that runs a path per thread (trace, shade, trace a shadow ray, next bounce) keeps a warp
// at every step until its slowest lane is through: on the Cornell box 6 of 32 lanes were active
// per instruction, in PSSMLT's chains 4.  Here each lane is a small state machine that always
// holds a walk (a closest hit or a shadow ray, of whatever bounce of whatever path), and the warp
// alternates two things:
//   * walk     the walking lanes vote on the kind of unit (TravVote) and the winners take one
//              step of their walk;
//   * service  once at most an eighth of the lanes still walk, every lane whose walk has ended is served
//              together: a shadow ray's answer is added, a hit is shaded, an ended path is handed
//              to the task and the lane's next path is begun, and the lane's next walk is set up.
// So a lane with a short path goes on to its next one instead of waiting, and both the walk and
// the shading run with most of the warp.  Each lane's sequence of walks, draws and float
// operations is that of the plain loop, so the results are too, bit for bit.
//
// A path's shadow term is evaluated when its light sample is (Ln, the radiance if the ray gets
// through) and the ray is traced only if it can change L (shadow_contributes).
//
// Task: what the paths are.  start(&ray, &smp) begins this lane's next path (false: none left),
// finish(L, smp) takes the radiance of the one that ended; both are called by the lanes concerned
// together.  hit(depth, found, h) and lit() hear of every closest hit and, for the vertex in
// task.vertex, of a shadow ray that got through (kRecord).  Smp is the task's sampler type.
//
// kRecord: the paths are to be replayed from those records (k_adjoint.cu), so a shadow ray is also
// traced when only the derivative of its term can be other than zero (Bounce::lit).
#pragma once
#include "dev_shading.cuh"

namespace bn {

// a warp's walking lanes step until at most `stop` of them still walk (every lane calls it)
template <int kAny, bool kWT, int kWalk, class Stack>
__device__ __forceinline__ void walk_down_to(int stop, Trav& tr, const DevScene& s, Stack& stk, TraceCounters* tc) {
  for (;;) {
    const TravVote v(0xffffffffu, true, tr.mode);
    if (v.walking() <= stop) break;
    if (tr.mode == v.pick()) trav_step<kAny, kWT, kWalk, 4, true>(tr, s, stk, tc);
  }
}

// Lanes of a warp that take paths: n paths spread over every warp of the grid when there are
// fewer of them than lanes (short renders are bound by the latency of one path's walks, which
// more warps with fewer lanes hide better).
__host__ __device__ __forceinline__ int machine_lanes(long long n, long long warps) {
  const long long l = (n + warps - 1) / warps;
  return l < 1 ? 1 : (l > 32 ? 32 : static_cast<int>(l));
}

// Launch shape.  Blocks of 128, 4 per SM (128 registers): 64 spp of the Cornell box / 32 spp of
// Cornell with objects / two instanced views of 4 spp took 10.0 / 45.7 / 35.8 ms, at 5 blocks 10.4 /
// 48.4 / 35.5, at 6 blocks 11.6 / 50.1 / 36.1 (spills), at 3 up to 15 % more than at 4.  Service when 8, 4, 3
// or 2 of the 32 lanes still walk: Cornell with objects at 3 spp 4.90 4.74 4.66 4.73 ms, one instanced
// view at 1 spp 6.33 6.34 6.49 6.76, 65,536 PSSMLT chains 55.1 53.0 52.5 52.9 (when 12 still walk 57): an
// eighth of the lanes.
constexpr int kMachineThreads = 128, kMachineBlocks = 4;
constexpr int kMachineRefill = 4;
constexpr int kMachineStack = 16;  // stack entries per lane in shared memory

enum : int { kLaneNew = 0, kLaneClosest = 1, kLaneShadow = 2, kLaneIdle = 3 };

template <bool kWT, int kWalk, bool kSimple, bool kFixed7, bool kRecord = false, class Task, class Smp>
__device__ __forceinline__ void path_machine(const DevScene& s, Task& task, Smp& smp, int max_depth, int rr_depth,
                                             int lanes) {
  static_assert(kWalk != kWalkCount, "counting walks run the plain loop");
  __shared__ int2 stack_block[kMachineStack * kMachineThreads];
  SharedStack<kMachineStack, kMachineThreads> stk(stack_block);
  TraceCounters tc{0, 0, 0};
  Trav tr;
  tr.mode = kTravDone;
  tr.any = false;
  int phase = static_cast<int>(threadIdx.x & 31) < lanes ? kLaneNew : kLaneIdle;
  V3 L = mk(0.f, 0.f, 0.f), Ln = L, beta = L, nd = L;
  float pdf = 0.f;
  int depth = 0;
  bool ends = false;
  for (;;) {
    const bool walking = tr.mode != kTravDone;
    // service every lane whose walk has ended
    if (!walking && phase != kLaneIdle) {
      bool over = false;
      V3 org = mk(0.f, 0.f, 0.f), dir = org;  // the next walk
      float tmax = CUDART_INF_F;
      if (phase == kLaneClosest) {
        if constexpr (kRecord) task.hit(depth, tr.found(), tr.hit());
        if (!tr.found()) {
          over = true;
        } else {
          Bounce b;
          PathState ps;
          ps.ray = tr.wr;
          ps.L = L;
          ps.beta = beta;
          ps.pdf_bsdf = pdf;
          ps.depth = depth;
          const int vertex = depth;
          bounce_shade<kFixed7, kSimple>(s, ps, tr.hit(), smp, max_depth, rr_depth, &b);
          L = ps.L;
          beta = ps.beta;
          pdf = ps.pdf_bsdf;
          depth = ps.depth;
          ends = b.ends;
          org = b.p;
          if (b.shadow || (kRecord && b.lit)) {
            if constexpr (kRecord) task.vertex = vertex;
            Ln = b.Ln;
            nd = ps.ray.d;
            dir = b.sh_d;
            tmax = b.sh_t;
            phase = kLaneShadow;
          } else {
            dir = ps.ray.d;
            over = ends;
          }
        }
      } else if (phase == kLaneShadow) {
        if (!tr.found()) {
          L = Ln;
          if constexpr (kRecord) task.lit();
        }
        org = tr.wr.o;
        dir = nd;
        phase = kLaneClosest;
        over = ends;
      }
      if (over) task.finish(L, smp);
      if (over || phase == kLaneNew) {
        Ray ray;
        if (task.start(&ray, &smp)) {
          org = ray.o;
          dir = ray.d;
          L = mk(0.f, 0.f, 0.f);
          beta = mk(1.f, 1.f, 1.f);
          pdf = 0.f;
          depth = 0;
          phase = kLaneClosest;
        } else {
          phase = kLaneIdle;
        }
      }
      if (phase != kLaneIdle) {
        Ray ray;
        ray.o = org;
        ray.d = dir;
        tr.any = phase == kLaneShadow;
        trav_init<kWalk>(tr, s, ray, tmax, &tc);  // may end at once (the root box missed)
      }
    }
    // walk until few lanes still do
    const unsigned busy = __ballot_sync(0xffffffffu, phase != kLaneIdle);
    if (!busy) break;
    walk_down_to<kAnyRuntime, kWT, kWalk>(__popc(busy) * kMachineRefill / 32, tr, s, stk, &tc);
  }
}

// a grid-wide counter handed out to the lanes that call together, one atomic per group
__device__ __forceinline__ unsigned long long claim_next(unsigned long long* counter) {
  const unsigned act = __activemask();
  const int lane = threadIdx.x & 31, leader = __ffs(act) - 1;
  unsigned long long base = 0;
  if (lane == leader) base = atomicAdd(counter, static_cast<unsigned long long>(__popc(act)));
  base = __shfl_sync(act, base, leader);
  return base + __popc(act & ((1u << lane) - 1u));
}

}  // namespace bn
