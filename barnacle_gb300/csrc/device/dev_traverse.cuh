// Two-level BVH traversal: TLAS -> PrimitiveInstance -> BLAS (included by dev_geometry.cuh).
//
// Order and culling are the reference's (Aggregate/BVH.fs:11-58, Primitive.fs:111-129,
// Mesh.fs:188-242): near child first (left when d[axis] > 0), the instances of a TLAS leaf in
// order, each instance's BLAS walked completely before the next, every box tested against the
// current t with tMin = 1e-3.  Changes of form keep the SIMT lanes together and the loads few:
//  * an interior node tests its children at once, enters the near one and pushes the far one
//    with its entry distance; on pop the far child is entered only if that distance is still
//    <= t, which is exactly the reference's box test at pop time (a box that passed with a
//    larger t passes with the current t iff its entry distance is <= t).
//  * the wide walk reads one 128-byte record per step that holds the two binary levels below
//    the node (its grandchildren, see dev_types.cuh) and tests the four boxes together.  It
//    visits them in the binary walk's order (near child's near child first, by the split axes
//    of the node and of each child) and stacks the hits that pass so that they pop in that
//    order.  Because a nested box passes whenever its parent box would with the same t, it
//    visits the same leaves in the same order with the same t as the binary walk.  A scene is
//    walked wide (kWalkWide) when the upload built records for it (large scenes; small BVHs gain
//    nothing from them).  The counting walk (kWalkCount) is always the binary one, so its counts
//    equal the reference's (the root plus both children of every entered interior node).
//  * the walk is a flat state machine: each step is one bounded unit of work (a node record or
//    pair, a leaf's triangles, a TLAS leaf's instances) at either BVH level, with pops folded
//    into the step that needs them, so lanes at different levels run the same loop body and
//    reconverge after every step instead of waiting out each other's nested BLAS loops.  A
//    caller can refill a lane with a new ray as soon as its walk finishes, and let only the
//    lanes at one kind of unit take a step (TravVote).

namespace bn {

// the slab test that also reports the entry distance max(1e-3, t0') used by the pop check
__device__ __forceinline__ bool box_hit_t(V3 bmin, V3 bmax, const Ray& r, V3 inv, float tmax_in, float* tentry) {
  const float t0x = __fmul_rn(__fsub_rn(bmin.x, r.o.x), inv.x), t1x = __fmul_rn(__fsub_rn(bmax.x, r.o.x), inv.x);
  const float t0y = __fmul_rn(__fsub_rn(bmin.y, r.o.y), inv.y), t1y = __fmul_rn(__fsub_rn(bmax.y, r.o.y), inv.y);
  const float t0z = __fmul_rn(__fsub_rn(bmin.z, r.o.z), inv.z), t1z = __fmul_rn(__fsub_rn(bmax.z, r.o.z), inv.z);
  // fminf/fmaxf give the same decisions as MinNative/MaxNative here: they differ only when t1 is
  // NaN (minps/maxps return t1), and such boxes are rejected by the NaN check anyway; the sign of
  // a zero cannot change max(1e-3, ...) <= min(t, ...)
  const float tmin = fmaxf(1e-3f, fmaxf(fminf(t0x, t1x), fmaxf(fminf(t0y, t1y), fminf(t0z, t1z))));
  const float tmax = fminf(tmax_in, fminf(fmaxf(t0x, t1x), fminf(fmaxf(t0y, t1y), fmaxf(t0z, t1z))));
  const bool nan = (t1x != t1x) | (t1y != t1y) | (t1z != t1z);
  *tentry = tmin;
  return (tmin <= tmax) & !nan;
}

enum : int { kTravNode = 0, kTravTri = 1, kTravInst = 2, kTravDone = 3 };

// the reference's near-child test d[axis] > 0 for the three axes at once (a zero or NaN component
// is not > 0, as in BVH.fs)
__device__ __forceinline__ int octant(V3 d) { return int(d.x > 0.f) | (int(d.y > 0.f) << 1) | (int(d.z > 0.f) << 2); }

// A walk's state.  The traversal kernels hold it in 64 to 80 registers with everything else, so what
// can be had from another field is not kept.
struct Trav {
  Ray wr;            // world ray
  V3 winv;
  Ray orr;           // the ray of the level: the object-space ray of the instance being walked, or wr
  V3 oinv;
  int ooct;          // octant of orr's direction: bit a set when d[a] > 0
  WtRay wt;
  float t;
  NodeRec n;         // current interior node of the binary walk (kTravNode), its box already passed
  int mode;
  int cur, base;     // node or record index, in the wide walk also the code of the BLAS leaf being
                     // processed; the level's base in nodes[] (binary walk)
  int tri_base;
  int sp, blas_sp0;  // blas_sp0: the stack below the BLAS being walked, -1 in the TLAS
  int ii, ii_end;    // instances of the TLAS leaf being processed; the BLAS walked is ii - 1's
  int ti, ti_end;    // triangles of the BLAS leaf being processed (binary walk)
  bool any;          // any-hit query (runtime choice, kAnyRuntime walks)
  // the hit at t: barycentrics, instance (-1: none), triangle or ~root of a sphere
  float hu, hv;
  int hinst, hprim;

  __device__ __forceinline__ bool found() const { return hinst >= 0; }
  __device__ __forceinline__ HitRec hit() const {
    HitRec h;
    h.t = t; h.u = hu; h.v = hv;
    h.inst = hinst;
    h.tri = hprim < 0 ? 0 : hprim;
    h.sphere_root = hprim < 0 ? ~hprim : 0;
    return h;
  }
};

// back to the TLAS with the world ray
__device__ __forceinline__ void trav_world(Trav& tr) {
  tr.orr = tr.wr;
  tr.oinv = tr.winv;
  tr.ooct = octant(tr.wr.d);
  tr.blas_sp0 = -1;
}

// enter a node whose box passed: an interior node is walked, a leaf's items are iterated
__device__ __forceinline__ void trav_enter(Trav& tr, int cur, const NodeRec& n) {
  tr.cur = cur;
  if (!n.leaf) {
    tr.n = n;
    tr.mode = kTravNode;
  } else if (tr.blas_sp0 < 0) {
    tr.ii = n.link;
    tr.ii_end = n.link + n.count;
    tr.mode = kTravInst;
  } else {
    tr.ti = n.link;
    tr.ti_end = n.link + n.count;
    tr.mode = kTravTri;
  }
}

// The walk's stack of far entries: a node or record index (or a leaf slot) with its entry
// distance.  LocalStack keeps them in the thread's local memory.  SharedStack keeps the bottom
// kShared entries in shared memory, one column per thread of a kBlock-thread block (lanes at
// different depths then fall on different banks), and the deeper ones in local memory, so the
// pushes and pops of a typical walk stay out of the L1 data cache the node loads use.
struct LocalStack {
  int sn[kStackSize];
  float st[kStackSize];
  __device__ __forceinline__ void put(int i, int n, float t) { sn[i] = n; st[i] = t; }
  __device__ __forceinline__ void get(int i, int* n, float* t) const { *n = sn[i]; *t = st[i]; }
};

template <int kShared, int kBlock>
struct SharedStack {
  using Entry = int2;
  int2* col;  // this thread's column of the block's kShared x kBlock array
  int sn[kStackSize - kShared];
  float st[kStackSize - kShared];
  __device__ __forceinline__ explicit SharedStack(int2* block_array) : col(block_array + threadIdx.x) {}
  __device__ __forceinline__ void put(int i, int n, float t) {
    if (i < kShared) {
      col[i * kBlock] = make_int2(n, __float_as_int(t));
    } else {
      sn[i - kShared] = n;
      st[i - kShared] = t;
    }
  }
  __device__ __forceinline__ void get(int i, int* n, float* t) const {
    if (i < kShared) {
      const int2 e = col[i * kBlock];
      *n = e.x;
      *t = __int_as_float(e.y);
    } else {
      *n = sn[i - kShared];
      *t = st[i - kShared];
    }
  }
};

// SharedStack without the distances, for any-hit walks: their t never shrinks, so that a box that
// passed still passes when it pops.
template <int kShared, int kBlock>
struct SharedCodes {
  using Entry = int;
  int* col;
  int sn[kStackSize - kShared];
  __device__ __forceinline__ explicit SharedCodes(int* block_array) : col(block_array + threadIdx.x) {}
  __device__ __forceinline__ void put(int i, int n, float) {
    if (i < kShared) col[i * kBlock] = n;
    else sn[i - kShared] = n;
  }
  __device__ __forceinline__ void get(int i, int* n, float* t) const {
    *n = i < kShared ? col[i * kBlock] : sn[i - kShared];
    *t = -CUDART_INF_F;
  }
};

// a leaf by its code in a wide record (dev_types.cuh): instances in the TLAS, triangles in a BLAS
__device__ __forceinline__ int leaf_code(const DevScene& s, int first, int count) {
  return ~((first << s.leaf_bits) | (count - 1));
}
__device__ __forceinline__ void leaf_items(const DevScene& s, int code, int* first, int* end) {
  *first = ~code >> s.leaf_bits;
  *end = *first + (~code & ((1 << s.leaf_bits) - 1)) + 1;
}
__device__ __forceinline__ void trav_enter_code(Trav& tr, const DevScene& s, int code) {
  if (tr.blas_sp0 < 0) {
    leaf_items(s, code, &tr.ii, &tr.ii_end);
    tr.mode = kTravInst;
  } else {
    tr.cur = code;
    tr.mode = kTravTri;
  }
}

__device__ __forceinline__ const float4* node4_at(const DevScene& s, int i) {
  return s.nodes4 + 8 * static_cast<size_t>(i);
}

// the next stacked node still within reach; an exhausted BLAS returns to the instances of its
// TLAS leaf, an exhausted TLAS ends the walk.  Binary entries are node indices within the level;
// wide entries are a record's slots: record indices (>= 0) or a leaf's code (< 0).
template <bool kWide, class Stack>
__device__ __forceinline__ void trav_pop(Trav& tr, const DevScene& s, const Stack& stk) {
  for (;;) {
    const int bottom = max(tr.blas_sp0, 0);
    while (tr.sp > bottom) {
      --tr.sp;
      int c;
      float te;
      stk.get(tr.sp, &c, &te);
      if (te <= tr.t) {
        if (!kWide) {
          trav_enter(tr, c, load_node(s.nodes, tr.base + c));
        } else if (c >= 0) {
          tr.cur = c;
          tr.mode = kTravNode;
        } else {
          trav_enter_code(tr, s, c);
        }
        return;
      }
    }
    if (tr.blas_sp0 >= 0) {
      tr.base = 0;
      trav_world(tr);
      if (tr.ii < tr.ii_end) {
        tr.mode = kTravInst;
        return;
      }
      continue;  // the TLAS leaf had no instance left: keep popping the TLAS
    }
    tr.mode = kTravDone;
    return;
  }
}

// kWalk: which walk and whether it counts its visits
enum : int { kWalkBinary = 0, kWalkCount = 1, kWalkWide = 2 };

template <int kWalk>
__device__ __forceinline__ void trav_init(Trav& tr, const DevScene& s, const Ray& ray, float tmax, TraceCounters* cnt) {
  tr.wr = ray;
  tr.winv = inv_dir(ray.d);
  tr.t = tmax;
  tr.hinst = -1;
  tr.sp = 0;
  tr.base = 0;
  tr.ii = tr.ii_end = 0;
  tr.ti = tr.ti_end = 0;
  trav_world(tr);
  const NodeRec root = load_node(s.nodes, 0);
  if (kWalk == kWalkCount) cnt->nodes++;
  float te;
  if (!box_hit_t(root.bmin, root.bmax, tr.wr, tr.winv, tr.t, &te)) {
    tr.mode = kTravDone;
  } else if (kWalk != kWalkWide || root.leaf) {
    trav_enter(tr, 0, root);
  } else {
    tr.cur = 0;  // the TLAS root's record
    tr.mode = kTravNode;
  }
}

// one wide step: the four slot boxes of record tr.cur; returns kStepPop when none is entered,
// kStepOverflow when the stack is full.  The slots are put in visit order by three conditional swaps
// (with the triangle test before a leaf's box test this took 6 instanced views of 4 spp from 95.3 to
// 90.8 ms; selecting each slot by its number cost twice the instructions)
// Without kOrdered (any-hit walks, whose answer no order changes and whose t never shrinks) the pair
// with the nearest slot comes first, in each pair the nearer slot, and nothing is stacked but the slots:
// the binary walk's order takes 25 instructions and 8 bytes per entry.  Binary order / no order /
// nearest pair first, kernel ms: six instanced views of 4 spp 77.6 / 79.6 / 77.2, Cornell with objects
// 17.42 / 16.95 / 16.91, material forward 11.52 / 11.19 / 11.20; 1,000,003 any hits among instances 0.636 / 0.642
// / 0.619, 131,071 in Cornell with objects 0.116 / 0.107 / 0.103.
enum : int { kStepOk = 0, kStepPop = 1, kStepOverflow = 2 };
template <bool kOrdered, class Stack>
__device__ __forceinline__ int trav_node4(Trav& tr, const DevScene& s, Stack& stk) {
  const Ray& r = tr.orr;
  const V3 inv = tr.oinv;
  const float4* q = node4_at(s, tr.cur);
  const float4 lx = __ldg(q), ly = __ldg(q + 1), lz = __ldg(q + 2);
  const float4 hx = __ldg(q + 3), hy = __ldg(q + 4), hz = __ldg(q + 5);
  const int4 ref = __ldg(reinterpret_cast<const int4*>(q + 6));
  int2 orders = make_int2(0, 0);
  if (kOrdered) orders = __ldg(reinterpret_cast<const int2*>(q + 7));
  float e0, e1, e2, e3;
  const bool h0 = box_hit_t(mk(lx.x, ly.x, lz.x), mk(hx.x, hy.x, hz.x), r, inv, tr.t, &e0);
  const bool h1 = box_hit_t(mk(lx.y, ly.y, lz.y), mk(hx.y, hy.y, hz.y), r, inv, tr.t, &e1);
  const bool h2 = box_hit_t(mk(lx.z, ly.z, lz.z), mk(hx.z, hy.z, hz.z), r, inv, tr.t, &e2);
  const bool h3 = box_hit_t(mk(lx.w, ly.w, lz.w), mk(hx.w, hy.w, hz.w), r, inv, tr.t, &e3);
  if (!(h0 | h1 | h2 | h3)) return kStepPop;
  // what a stack entry says of each slot: a record, a leaf's code, or nothing entered (no leaf has
  // that code)
  constexpr int kNone = static_cast<int>(0x80000000u);
  const int c0 = h0 ? ref.x : kNone, c1 = h1 ? ref.y : kNone, c2 = h2 ? ref.z : kNone, c3 = h3 ? ref.w : kNone;
  if (!kOrdered) {
    // (the entry distances are not negative, so their bits order as they do)
    const int f0 = h0 ? __float_as_int(e0) : 0x7fffffff, f1 = h1 ? __float_as_int(e1) : 0x7fffffff;
    const int f2 = h2 ? __float_as_int(e2) : 0x7fffffff, f3 = h3 ? __float_as_int(e3) : 0x7fffffff;
    const bool s01 = f1 < f0, s23 = f3 < f2, sp = min(f2, f3) < min(f0, f1);
    const int a = s01 ? c1 : c0, b = s01 ? c0 : c1, c = s23 ? c3 : c2, d = s23 ? c2 : c3;
    const int next = sp ? c : a, w1 = sp ? d : b, w2 = sp ? a : c, w3 = sp ? b : d;
    if (tr.sp + 3 > s.stack_cap && tr.sp + int(h0) + int(h1) + int(h2) + int(h3) - 1 > s.stack_cap) return kStepOverflow;
    if (w3 != kNone) stk.put(tr.sp++, w3, 0.f);
    if (w2 != kNone) stk.put(tr.sp++, w2, 0.f);
    if (w1 != kNone) stk.put(tr.sp++, w1, 0.f);
    if (next >= 0) tr.cur = next;
    else trav_enter_code(tr, s, next);
    return kStepOk;
  }
  // the binary walk's order (the near child's slots, then the far child's, each pair ordered by
  // that child's own split axis: BVH.fs near-child rule at both levels) depends on the ray only
  // through its octant; the upload stored the slot order of each octant, 8 bits per octant: bit 1
  // swaps the pairs, bits 0 and 4 the slots of the pair then first and second
  const int oct = tr.ooct;
  const unsigned order = static_cast<unsigned>(oct & 4 ? orders.y : orders.x) >> (8 * (oct & 3));
  const bool sp = order & 2u, sa = order & 1u, sb = order & 16u;
  const int a0 = sp ? c2 : c0, a1 = sp ? c3 : c1, b0 = sp ? c0 : c2, b1 = sp ? c1 : c3;
  const float ea0 = sp ? e2 : e0, ea1 = sp ? e3 : e1, eb0 = sp ? e0 : e2, eb1 = sp ? e1 : e3;
  const int v0 = sa ? a1 : a0, v1 = sa ? a0 : a1, v2 = sb ? b1 : b0, v3 = sb ? b0 : b1;
  const float t1 = sa ? ea0 : ea1, t2 = sb ? eb1 : eb0, t3 = sb ? eb0 : eb1;
  // the first slot entered comes next; the later ones are stacked to pop in order
  const bool p0 = v0 != kNone, p1 = v1 != kNone, p2 = v2 != kNone, p3 = v3 != kNone;
  if (tr.sp + 3 > s.stack_cap && tr.sp + int(p0) + int(p1) + int(p2) + int(p3) - 1 > s.stack_cap) return kStepOverflow;
  if (p3 && (p0 | p1 | p2)) stk.put(tr.sp++, v3, t3);
  if (p2 && (p0 | p1)) stk.put(tr.sp++, v2, t2);
  if (p1 && p0) stk.put(tr.sp++, v1, t1);
  const int next = p0 ? v0 : (p1 ? v1 : (p2 ? v2 : v3));
  if (next >= 0) tr.cur = next;
  else trav_enter_code(tr, s, next);
  return kStepOk;
}

// one step: a wide record or a node pair, one instance (kInstRun: the leaf's instances until one
// is entered), or kTris triangles of a leaf (0 = the rest of it); returns true once the walk is
// finished (tr.found() and tr.hit() give the answer).
// kAny: kClosest, kAnyHit, or kAnyRuntime (tr.any decides).  Every branch that exhausts its unit
// asks for a pop, which runs once at the end of the step.
enum : int { kClosest = 0, kAnyHit = 1, kAnyRuntime = 2 };
template <int kAny, bool kWT, int kWalk, int kTris = 1, bool kInstRun = false, class Stack>
__device__ __forceinline__ bool trav_step(Trav& tr, const DevScene& s, Stack& stk, TraceCounters* cnt) {
  constexpr bool kCount = kWalk == kWalkCount, kWide = kWalk == kWalkWide;
  const bool any = kAny == kAnyRuntime ? tr.any : kAny == kAnyHit;
  bool pop = false;
  if (kWide && tr.mode == kTravNode) {
    const int r = trav_node4<kAny != kAnyHit>(tr, s, stk);

    if (r == kStepOverflow) {
      flag_error(s, BN_DEVERR_STACK_OVERFLOW);
      tr.mode = kTravDone;
      return true;
    }
    pop = r == kStepPop;
  } else if (tr.mode == kTravNode) {
    const Ray& r = tr.orr;
    const V3 inv = tr.oinv;
    const int li = tr.cur + 1, ri = tr.n.link;
    const NodeRec a = load_node(s.nodes, tr.base + li);
    const NodeRec b = load_node(s.nodes, tr.base + ri);
    if (kCount) cnt->nodes += 2;
    float ta, tb;
    const bool ha = box_hit_t(a.bmin, a.bmax, r, inv, tr.t, &ta);
    const bool hb = box_hit_t(b.bmin, b.bmax, r, inv, tr.t, &tb);
    const bool left_first = comp(r.d, tr.n.axis) > 0.f;
    if (ha && hb) {
      if (tr.sp >= s.stack_cap) {
        flag_error(s, BN_DEVERR_STACK_OVERFLOW);
        tr.mode = kTravDone;
        return true;
      }
      if (left_first) { stk.put(tr.sp, ri, tb); ++tr.sp; trav_enter(tr, li, a); }
      else { stk.put(tr.sp, li, ta); ++tr.sp; trav_enter(tr, ri, b); }
    } else if (ha) {
      trav_enter(tr, li, a);
    } else if (hb) {
      trav_enter(tr, ri, b);
    } else {
      pop = true;
    }
  } else if (tr.mode == kTravTri) {
    // kTris triangles of a BLAS leaf (0: the rest of the leaf): each the triangle test, then its AABB
    // test (Mesh.fs:204,231).  The reference tests the box first; a hit needs both, and the triangle
    // test turns most triangles away earlier.
    int done = 0, ti = tr.ti, ti_end = tr.ti_end;
    if (kWide) leaf_items(s, tr.cur, &ti, &ti_end);
#pragma unroll 1
    while (ti < ti_end) {
      const int j = ti++;
      const float4* tp = s.tris + 3 * (tr.tri_base + j);
      const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
      if (kCount) cnt->tris++;
      const V3 p0 = xyz(a), p1 = xyz(b), p2 = xyz(c);
      float tt, uu, vv;
      const bool h = kWT ? tri_wt(p0, p1, p2, tr.orr, tr.wt, tr.t, &tt, &uu, &vv)
                         : tri_mt(p0, p1, p2, tr.orr, tr.t, &tt, &uu, &vv);
      if (h) {
        const V3 lo = min_native(min_native(p0, p1), p2), hi = max_native(max_native(p0, p1), p2);
        if (box_hit(lo, hi, tr.orr, tr.oinv, tr.t)) {
          tr.hinst = tr.ii - 1;
          if (any) {
            tr.mode = kTravDone;
            return true;
          }
          tr.t = tt;
          tr.hprim = j; tr.hu = uu; tr.hv = vv;
        }
      }
      if (kTris > 0 && ++done >= kTris) break;
    }
    pop = ti >= ti_end;
    if (!kWide) tr.ti = ti;
    else if (!pop) tr.cur = leaf_code(s, ti, ti_end - ti);
  } else if (tr.mode == kTravInst) {
    // the next instance of a TLAS leaf, or with kInstRun the leaf's instances until one is
    // entered (PrimitiveInstance.Intersect, Primitive.fs:111-129)
    bool entered = false;
#pragma unroll 1
    while (!entered && tr.ii < tr.ii_end) {
      const int k = tr.ii++;
      const DevInstance* I = s.inst + k;
      if (kCount) cnt->insts++;
      // the instance's first line in eight independent loads: bounds, WorldToObject, the BLAS
      // root's box and the indices, so one memory round trip serves the whole visit
      const float4* line = reinterpret_cast<const float4*>(I);
      const float4 bmin = __ldg(line), bmax = __ldg(line + 1);
      float4 w2o[3];
      w2o[0] = __ldg(line + 2); w2o[1] = __ldg(line + 3); w2o[2] = __ldg(line + 4);
      const float4 rlo = __ldg(line + 5), rhi = __ldg(line + 6);
      const int4 ids = __ldg(reinterpret_cast<const int4*>(line + 7));  // prim_type, node_base, tri_base, node4_root
      if (box_hit(xyz(bmin), xyz(bmax), tr.wr, tr.winv, tr.t)) {
        Ray orr;
        orr.o = xf_point(w2o, tr.wr.o);
        orr.d = xf_dir(w2o, tr.wr.d);
        if (ids.x == kPrimSphere) {
          float ts;
          const int root = sphere_hit(bmax.w, orr, tr.t, &ts);
          if (root) {
            tr.hinst = k;
            if (any) {
              tr.mode = kTravDone;
              return true;
            }
            tr.t = ts;
            tr.hprim = ~root; tr.hu = 0.f; tr.hv = 0.f;
          }
        } else {
          const V3 oinv = inv_dir(orr.d);
          auto enter = [&]() {
            tr.orr = orr;
            tr.oinv = oinv;
            tr.ooct = octant(orr.d);
            if (kWT) tr.wt = wt_setup(orr.d);
          };
          const int base = ids.y;
          float te;
          if (kWide && ids.w >= 0) {
            // the root's box from the instance line, its record next (the root is interior)
            if (box_hit_t(xyz(rlo), xyz(rhi), orr, oinv, tr.t, &te)) {
              enter();
              tr.base = base;
              tr.tri_base = ids.z;
              tr.blas_sp0 = tr.sp;
              tr.cur = ids.w;
              tr.mode = kTravNode;
              entered = true;
            }
          } else {
            const NodeRec root = load_node(s.nodes, base);
            if (kCount) cnt->nodes++;
            if (box_hit_t(root.bmin, root.bmax, orr, oinv, tr.t, &te)) {
              enter();
              tr.base = base;
              tr.tri_base = ids.z;
              tr.blas_sp0 = tr.sp;
              if (kWide) trav_enter_code(tr, s, leaf_code(s, root.link, root.count));  // (a leaf)
              else trav_enter(tr, 0, root);
              entered = true;
            }
          }
        }
      }
      if (!kInstRun) break;
    }
    pop = !entered && tr.ii >= tr.ii_end;
  }
  if (pop) trav_pop<kWide>(tr, s, stk);
  return tr.mode == kTravDone;
}

// Lanes of a warp at different kinds of unit (a node record, a leaf's triangles, instances) run
// different branches of a step one after the other, each with its own chain of dependent loads.
// With a vote only the lanes in the mode with the largest weighted count take the step (instances
// weigh 3, nodes and triangles 2); the others keep their state and wait.  Each lane's sequence of
// units is unchanged, so its result is too.  The vote is two ballots on the mode's bits, which also
// tell how many lanes still walk; a lane that does not counts as done (both bits).
struct TravVote {
  unsigned act, b0, b1;
  __device__ __forceinline__ TravVote(unsigned lanes, bool walking, int mode) : act(lanes) {
    static_assert(kTravNode == 0 && kTravTri == 1 && kTravInst == 2 && kTravDone == 3, "mode bits");
    b0 = __ballot_sync(act, !walking || (mode & 1));
    b1 = __ballot_sync(act, !walking || (mode & 2));
  }
  __device__ __forceinline__ int walking() const { return __popc(act & ~(b0 & b1)); }
  __device__ __forceinline__ int pick() const {
    const int cn = 2 * __popc(act & ~(b0 | b1));
    const int ct = 2 * __popc(b0 & ~b1);
    const int ci = 3 * __popc(b1 & ~b0);
    return (cn >= ct && cn >= ci) ? kTravNode : (ct >= ci ? kTravTri : kTravInst);
  }
};

// A walk, inlined at its call site with the query fixed at compile time.
template <int kAny, bool kWT, int kWalk>
__device__ __forceinline__ bool trace_walk_inline(const DevScene& s, const Ray& ray, float tmax, HitRec* hit,
                                                  TraceCounters* cnt) {
  LocalStack stk;
  Trav tr;
  trav_init<kWalk>(tr, s, ray, tmax, cnt);
  while (!trav_step<kAny, kWT, kWalk, 0>(tr, s, stk, cnt)) {
  }
  if (kAny == kClosest) *hit = tr.hit();
  return tr.found();
}

// One walk for both queries, kept out of line: a path loop that traces closest and any hits
// then holds a single copy of the traversal code.  That keeps a large kernel whose time goes to
// shading within the instruction cache; a kernel whose time goes to long walks keeps them
// inlined, where the walk's registers are allocated with the loop around it.
template <bool kWT, int kWalk>
__device__ __noinline__ bool trace_walk_outline(const DevScene& s, const Ray& ray, float tmax, bool any, HitRec* hit,
                                                TraceCounters* cnt) {
  LocalStack stk;
  Trav tr;
  tr.any = any;
  trav_init<kWalk>(tr, s, ray, tmax, cnt);
  while (!trav_step<kAnyRuntime, kWT, kWalk, 0>(tr, s, stk, cnt)) {
  }
  if (!any) *hit = tr.hit();
  return tr.found();
}

template <bool kWT, int kWalk, bool kOutline = false>
__device__ __forceinline__ bool trace_closest(const DevScene& s, const Ray& ray, float tmax, HitRec* hit, TraceCounters* cnt) {
  if (kOutline) return trace_walk_outline<kWT, kWalk>(s, ray, tmax, false, hit, cnt);
  return trace_walk_inline<kClosest, kWT, kWalk>(s, ray, tmax, hit, cnt);
}

template <bool kWT, int kWalk, bool kOutline = false>
__device__ __forceinline__ bool trace_any(const DevScene& s, const Ray& ray, float tmax, TraceCounters* cnt) {
  HitRec h;
  if (kOutline) return trace_walk_outline<kWT, kWalk>(s, ray, tmax, true, &h, cnt);
  return trace_walk_inline<kAnyHit, kWT, kWalk>(s, ray, tmax, &h, cnt);
}

}  // namespace bn
