// svo_trace.cuh - device code of the sparse-voxel-octree first-hit ray cast
// for sm_103a (included by svo_kernels.cu and svo_noalloc.cu).
//
// One persistent kernel per frame: ray generation (RendererBase::InitRayDir /
// RenderRect, cell/renderer_base.h:50-61, cell/ppu_renderer.cpp:43-70),
// octree descent (RecTrace, cell/ppu_renderer.cpp:18-41, with FindFirstChild
// and GoNext of cell/spu/trace_spu.cpp:48-93), Lambert shading and an
// optional hard-shadow ray per hit, fused.
//
// Design (GB300):
//  * persistent grid (SMs x resident blocks).  Every lane runs its own small
//    state machine (primary ray -> shadow ray -> idle) one traversal step per
//    loop iteration; idle lanes of a warp are refilled together from a
//    global ray counter (one atomic per refill), so a warp never waits for
//    the slowest ray of a tile and the shadow rays of some lanes overlap the
//    primary rays of others.  Consecutive ray ids map to 8x4 pixel tiles, so
//    lanes refilled together trace neighbouring pixels;
//  * node records are 8 B, four to an L2 sector: the record of the first
//    child and a nibble per child that tells node, leaf and null apart.  A
//    ray reads a record when it enters (or returns to) a node and keeps it in
//    two registers, so a step over a null child reads no memory.  Against
//    32-byte records of 8 child words read at every step (2048^3 terrain,
//    1920x1080, shadow rays): with the updates below 598 -> 524 us, a
//    160x120 frame 71 -> 60 us; bit masks and a popcount in place of the
//    nibbles cost more than the loads saved (575 us).
//    Staging the breadth-first first `smem_nodes` records (the top tree
//    levels) in shared memory is a separately compiled variant the launch
//    configuration can ask for; reading every record through L1 measured as
//    fast or faster, so it is off by default;
//  * the recursion of RecTrace becomes an explicit per-lane stack of
//    (node id, child, slab box) frames, so a pop restores the parent's exact
//    float values: every operation is an explicit round-to-nearest intrinsic
//    (no FMA contraction), which keeps hit ids bit-identical to the FP32
//    restatement of the reference;
//  * every loop is bounded: a ray that exceeds the step cap or the stack
//    depth stops, is reported as a miss and sets a status bit;
//  * an optional frame time budget bounds the queue itself: a warp about to
//    take new rays after the budget has elapsed (the global timer against
//    its block's start) takes none, and the frame reports a timeout.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "yv_internal.h"
#include "yv_kernels.h"

namespace yv {
namespace {

constexpr uint32_t kFetchCap = 1u << 20;
// Traversal steps between two warp votes (refill / end-of-ray handling): a vote
// and a pass through the end of a ray cost every lane of the warp, a lane whose
// ray has ended waits for the rest of its group.  1920x1080 frame with shadow
// rays / 160x120 / 641x479 with the detail cut-off: 512 / 50.5 / 96.5 us at 8
// steps, 502 / 49.3 / 93.7 at 24, 512 / 49.3 / 93.8 at 48.  Unrolled 6 deep
// (504 us at 4): more copies overflow the instruction cache.
constexpr int kStepsPerVote = 24;

struct Box {
  float x1, y1, z1, x2, y2, z2;
};

__device__ __forceinline__ float max3f(float a, float b, float c) {
  float m = a > b ? a : b;  // max_vec_float3 order
  return m > c ? m : c;
}
// Minimum / maximum for the comparisons of the traversal (slab values are
// never NaN; +0 and -0 compare equal, so the choice between them is moot).
__device__ __forceinline__ float fmin3(float a, float b, float c) {
  float m;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
  return m;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float m;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
  return m;
}

// FindFirstChild (cell/spu/trace_spu.cpp:48-68).  The traversal is bound by
// the half-rate ALU pipe (compares, selects, logic), so the box updates here
// and in `advance` are written as predicated moves and FP32 adds, which the
// compiler's selects would put on that pipe.
__device__ __forceinline__ uint32_t ffc(Box& t) {
  const float te = fmax3(t.x1, t.y1, t.z1);
  uint32_t ch;
  // te > 0.5 (x1 + x2) as 2 te > x1 + x2 (both scalings by two are exact), so
  // that the halving is the predicated write itself
  asm("{\n\t.reg .pred px, py, pz;\n\t.reg .f32 mx, my, mz, t2;\n\t"
      "add.rn.f32 mx, %1, %4;\n\tadd.rn.f32 my, %2, %5;\n\tadd.rn.f32 mz, %3, %6;\n\t"
      "add.rn.f32 t2, %7, %7;\n\t"
      "setp.gt.f32 px, t2, mx;\n\tsetp.gt.f32 py, t2, my;\n\tsetp.gt.f32 pz, t2, mz;\n\t"
      "@px mul.rn.f32 %1, mx, 0f3F000000;\n\t@!px mul.rn.f32 %4, mx, 0f3F000000;\n\t"
      "@py mul.rn.f32 %2, my, 0f3F000000;\n\t@!py mul.rn.f32 %5, my, 0f3F000000;\n\t"
      "@pz mul.rn.f32 %3, mz, 0f3F000000;\n\t@!pz mul.rn.f32 %6, mz, 0f3F000000;\n\t"
      "selp.u32 %0, 4, 0, px;\n\t@py or.b32 %0, %0, 8;\n\t@pz or.b32 %0, %0, 16;\n\t}"
      : "=&r"(ch), "+f"(t.x1), "+f"(t.y1), "+f"(t.z1), "+f"(t.x2), "+f"(t.y2), "+f"(t.z2)
      : "f"(te));
  return ch;
}

// GoNext (cell/spu/trace_spu.cpp:70-93) in two parts: the exit axis (the
// argmin tie order of :75-78) as the child bit it flips, and the move into
// the sibling across it.
__device__ __forceinline__ uint32_t exit_bit(const Box& t) {
  // z where z2 <= min(x2, y2), else x where x2 <= y2: the minimum, which the
  // step needs anyway, in place of three chained compares (523 -> 514 us)
  const float m = fmin3(t.x2, t.y2, t.z2);
  return t.z2 == m ? 16u : (t.x2 == m ? 4u : 8u);
}

// On the crossed axis t1, t2 <- t2, t2 + (t2 - t1); predicated, the lanes of
// a warp cross different axes.
__device__ __forceinline__ void advance(uint32_t& ch, Box& t, uint32_t bit) {
  ch ^= bit;
  asm("{\n\t.reg .pred px, py, pz;\n\t.reg .f32 dx, dy, dz;\n\t"
      "setp.eq.u32 px, %6, 4;\n\tsetp.eq.u32 py, %6, 8;\n\tsetp.eq.u32 pz, %6, 16;\n\t"
      "sub.rn.f32 dx, %3, %0;\n\tsub.rn.f32 dy, %4, %1;\n\tsub.rn.f32 dz, %5, %2;\n\t"
      "@px mov.f32 %0, %3;\n\t@py mov.f32 %1, %4;\n\t@pz mov.f32 %2, %5;\n\t"
      "@px add.rn.f32 %3, %3, dx;\n\t@py add.rn.f32 %4, %4, dy;\n\t"
      "@pz add.rn.f32 %5, %5, dz;\n\t}"
      : "+f"(t.x1), "+f"(t.y1), "+f"(t.z1), "+f"(t.x2), "+f"(t.y2), "+f"(t.z2)
      : "r"(bit));
}

// Child word c of node id of a caller's pool, whose flags word is fl: the
// reference's 40-byte VoxNode {flags, data, child[8]} read in place, its leaf
// and null children folded into one encoding (a child is null by its word,
// whatever the flags say).
__device__ __forceinline__ uint32_t ref_child_word(const SvoDeviceScene& sc, uint32_t id,
                                                   uint32_t fl, uint32_t c) {
  const uint32_t cw =
      __ldg(reinterpret_cast<const uint32_t*>(sc.nodes) + 10 * (size_t)id + 2 + c);
  return ((fl >> c) & 1u) ? (YV_DW_LEAF | cw) : ((cw & 0x80000000u) ? YV_DW_NULL : cw);
}

// Nanoseconds of the GPU's global timer.
__device__ __forceinline__ unsigned long long global_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// One stack frame: a level whose current child still has a next sibling
// along the ray - the node, the child taken and that child's slab box,
// exactly as RecTrace holds them in its activation record - and the level.
// Levels whose current child is the last one the ray crosses are never
// pushed: returning to them would only return further.
struct __align__(16) Frame {
  uint32_t node;
  float x1, y1, z1;
  float x2, y2, z2;
  uint32_t chlev;  // child (x 4) | level << 8
};

enum : uint32_t { kIdle = 0, kPrimary = 1, kShadow = 2, kDone = 3 };
enum : int { kContinue = 0, kHit = 1, kMiss = 2 };
// trace_step's `leaf` for a leaf child of the library's layout: its attribute
// is looked up once, at the end of the ray (hit_leaf)
constexpr uint32_t kLeafOfNode = 0xFFFFFFFFu;

// Traversal state of one lane.
struct Trace {
  // current child and direction mirror, both x 4: bits 2, 3 and 4 for x, y, z
  uint32_t node, ch, df, fetches;
  // the node's record (first node child, child codes); a caller's VoxNode:
  // its flags
  uint32_t first, codes;
  uint32_t sp;  // frames held
  uint32_t lo;  // with a shared-memory ring: frames below lo are in local memory
  int level;
  Box t;
};

// Per-lane frame stack.  kRing = 0: every frame in a local-memory array.
// kRing > 0 (a power of two): the newest kRing frames in a shared-memory
// ring, one 16-byte column per lane (lane-contiguous, so a warp's stores and
// loads are conflict-free and move only the active lanes' bytes); a push
// into a full ring first moves the oldest frame to the local array.
template <int kRing>
__device__ __forceinline__ void push_frame(Frame* stk, uint4* ring, Trace& tr, const Frame& f) {
  if (kRing == 0) {
    stk[tr.sp++] = f;
    return;
  }
  if (tr.sp - tr.lo == (uint32_t)kRing) {
    const uint32_t s = tr.lo & (uint32_t)(kRing - 1);
    const uint4 q0 = ring[(2 * s) * 32], q1 = ring[(2 * s + 1) * 32];
    Frame g;
    g.node = q0.x;
    g.x1 = __uint_as_float(q0.y); g.y1 = __uint_as_float(q0.z); g.z1 = __uint_as_float(q0.w);
    g.x2 = __uint_as_float(q1.x); g.y2 = __uint_as_float(q1.y); g.z2 = __uint_as_float(q1.z);
    g.chlev = q1.w;
    stk[tr.lo++] = g;
  }
  const uint32_t s = tr.sp & (uint32_t)(kRing - 1);
  ring[(2 * s) * 32] =
      make_uint4(f.node, __float_as_uint(f.x1), __float_as_uint(f.y1), __float_as_uint(f.z1));
  ring[(2 * s + 1) * 32] =
      make_uint4(__float_as_uint(f.x2), __float_as_uint(f.y2), __float_as_uint(f.z2), f.chlev);
  ++tr.sp;
}

template <int kRing>
__device__ __forceinline__ Frame pop_frame(const Frame* stk, const uint4* ring, Trace& tr) {
  --tr.sp;
  if (kRing == 0) return stk[tr.sp];
  if (tr.sp < tr.lo) {
    tr.lo = tr.sp;
    return stk[tr.sp];
  }
  const uint32_t s = tr.sp & (uint32_t)(kRing - 1);
  const uint4 q0 = ring[(2 * s) * 32], q1 = ring[(2 * s + 1) * 32];
  Frame g;
  g.node = q0.x;
  g.x1 = __uint_as_float(q0.y); g.y1 = __uint_as_float(q0.z); g.z1 = __uint_as_float(q0.w);
  g.x2 = __uint_as_float(q1.x); g.y2 = __uint_as_float(q1.y); g.z2 = __uint_as_float(q1.z);
  g.chlev = q1.w;
  return g;
}


// Reads what the traversal keeps of the node tr.node.
// kStaged: the first nsm records are read from shared memory.
template <bool kRef, bool kStaged>
__device__ __forceinline__ void enter_node(const SvoDeviceScene& sc, const uint32_t* sm,
                                           uint32_t nsm, Trace& tr) {
  if (kRef) {
    tr.codes = __ldg(reinterpret_cast<const uint32_t*>(sc.nodes) + 10 * (size_t)tr.node);
    return;
  }
  const uint2 v = (kStaged && tr.node < nsm)
                      ? reinterpret_cast<const uint2*>(sm)[tr.node]
                      : __ldg(reinterpret_cast<const uint2*>(sc.nodes) + tr.node);
  tr.first = v.x;
  tr.codes = v.y;
}

// SetupTrace (reaction/report/voxel.tex:312-326) + RecTrace entry test
// (cell/ppu_renderer.cpp:20-21) + the root fetch.  False: the ray misses.
template <bool kRef = false, bool kStaged = false>
__device__ __forceinline__ bool begin_trace(const SvoDeviceScene& sc, const uint32_t* sm,
                                            uint32_t nsm, float px, float py, float pz,
                                            float dx, float dy, float dz, Trace& tr,
                                            uint32_t& err) {
  uint32_t df = 0;
  if (dx < 0.f) { px = __fsub_rn(1.f, px); dx = -dx; df |= 4u; }
  if (dy < 0.f) { py = __fsub_rn(1.f, py); dy = -dy; df |= 8u; }
  if (dz < 0.f) { pz = __fsub_rn(1.f, pz); dz = -dz; df |= 16u; }
  Box R;
  R.x1 = __fdiv_rn(__fsub_rn(0.f, px), dx);
  R.x2 = __fdiv_rn(__fsub_rn(1.f, px), dx);
  R.y1 = __fdiv_rn(__fsub_rn(0.f, py), dy);
  R.y2 = __fdiv_rn(__fsub_rn(1.f, py), dy);
  R.z1 = __fdiv_rn(__fsub_rn(0.f, pz), dz);
  R.z2 = __fdiv_rn(__fsub_rn(1.f, pz), dz);
  tr.fetches = 0;
  if (!(fmax3(R.x1, R.y1, R.z1) < fmin3(R.x2, R.y2, R.z2))) return false;
  const uint32_t root = sc.root_word;
  if ((root & (YV_DW_NULL | YV_DW_LEAF)) || fmin3(R.x2, R.y2, R.z2) <= 0.f) return false;
  if (root >= sc.n_nodes) {
    err |= YV_DEV_ERR_POOL;
    return false;
  }
  tr.node = root;
  tr.df = df;
  tr.level = 0;
  tr.sp = 0;
  tr.lo = 0;
  tr.fetches = 1;
  enter_node<kRef, kStaged>(sc, sm, nsm, tr);
  tr.t = R;
  tr.ch = ffc(tr.t);
  return true;
}

// What the ray may do at its current child: the child ahead of the ray's
// origin (or, for a primary ray, a leaf behind it) is a hit or a descent, any
// other is passed over.
struct Probe {
  bool leaf;   // a leaf child (else a node where `take` is set)
  bool take;   // the ray hits it or descends into it
  uint32_t w;  // the node child's code in the top nibble; caller's pool: the
               // child word
};

template <bool kRef>
__device__ __forceinline__ Probe probe_child(const SvoDeviceScene& sc, const Trace& tr,
                                             bool cull) {
  Probe p;
  const uint32_t c = tr.ch ^ tr.df;
  const bool ahead = fmin3(tr.t.x2, tr.t.y2, tr.t.z2) > 0.f;
  if (kRef) {
    p.w = ref_child_word(sc, tr.node, tr.codes, c >> 2);
    p.leaf = (p.w & YV_DW_LEAF) != 0u;
    p.take = p.leaf ? (!cull || ahead) : (!(p.w & YV_DW_NULL) && ahead);
  } else {
    p.w = tr.codes << c;
    p.leaf = p.w >= (YV_CODE_LEAF << 28);
    p.take = (ahead || (p.leaf && !cull)) && (p.leaf || (int32_t)p.w >= 0);
  }
  return p;
}

// One step of RecTrace: test the current child (leaf -> hit, subtree ->
// descend), else move to the next sibling, first returning to the nearest
// pushed level when this one is exhausted (that level's next sibling exists
// by construction, so both cases share the move).
// kRef (caller-supplied VoxNode pool): child refs are range-checked, depth
// is capped at YV_MAX_DEPTH levels and a ray stops with YV_DEV_ERR_ITER after
// kFetchCap fetches.  The library's own layout is validated acyclic, in
// range and at most YV_MAX_DEPTH levels deep when it is built, so it needs
// none of these.  In both cases a push happens at level < YV_MAX_DEPTH - 1,
// so at most YV_MAX_DEPTH - 1 frames are ever held.
// kLod (library layout only): before descending into a subtree whose cube
// side 2^-(level+1) is smaller than max(t_enter, 0) * lod_coef, the ray stops
// there as at a leaf, with the subtree's level-of-detail attribute.
// kShared (library layout only): the scene may have a table of children
// (sc.child).  Compiled out elsewhere: the test alone, of a kernel parameter at
// each descent, took a 1920x1080 frame 563 -> 574 us and 641x479 with the detail
// cut-off 93.6 -> 97.5.
template <bool kRef, int kRing, bool kStaged = false, bool kLod = false, bool kShared = false>
__device__ __forceinline__ int trace_step(const SvoDeviceScene& sc, const uint32_t* sm,
                                          uint32_t nsm, Frame* stk, uint4* ring, Trace& tr,
                                          bool cull, uint32_t& leaf, uint32_t& err,
                                          float lod_coef = 0.f) {
  const Probe p = probe_child<kRef>(sc, tr, cull);
  // exit axis of the current child and whether it is the last one along
  // the ray in this node (needed by both the descent and the sibling move)
  uint32_t e = exit_bit(tr.t);
  const bool last = (tr.ch & e) != 0u;
  if (p.take) {
    if (p.leaf) {
      leaf = kRef ? (p.w & 0x7FFFFFFFu) : kLeafOfNode;
      return kHit;
    }
    uint32_t w = kRef ? p.w : tr.first + (p.w >> 28);
    if (kShared && sc.child) w = __ldg(sc.child + w);
    if (kLod) {
      const float side = __int_as_float((126 - tr.level) << 23);  // 2^-(level+1)
      const float te = fmaxf(fmax3(tr.t.x1, tr.t.y1, tr.t.z1), 0.f);
      if (side < __fmul_rn(te, lod_coef)) {
        leaf = __ldg(sc.node_data + w);
        return kHit;
      }
    }
    // descend: the recursive call of cell/ppu_renderer.cpp:34
    if (kRef) {
      if (tr.fetches >= kFetchCap) {
        err |= YV_DEV_ERR_ITER;
        return kMiss;
      }
      if (tr.level + 1 >= YV_MAX_DEPTH) {
        err |= YV_DEV_ERR_DEPTH;
        return kMiss;
      }
      if (w >= sc.n_nodes) {
        err |= YV_DEV_ERR_POOL;
        return kMiss;
      }
    }
    ++tr.fetches;
    if (!last) {
      Frame f;
      f.node = tr.node;
      f.x1 = tr.t.x1; f.y1 = tr.t.y1; f.z1 = tr.t.z1;
      f.x2 = tr.t.x2; f.y2 = tr.t.y2; f.z2 = tr.t.z2;
      f.chlev = tr.ch | ((uint32_t)tr.level << 8);
      push_frame<kRing>(stk, ring, tr, f);
    }
    ++tr.level;
    tr.node = w;
    enter_node<kRef, kStaged>(sc, sm, nsm, tr);
    tr.ch = ffc(tr.t);
    return kContinue;
  }
  if (last) {
    if (tr.sp == 0) return kMiss;
    const Frame f = pop_frame<kRing>(stk, ring, tr);
    tr.node = f.node;
    enter_node<kRef, kStaged>(sc, sm, nsm, tr);
    tr.ch = f.chlev & 0xFFu;
    tr.level = (int)(f.chlev >> 8);
    tr.t.x1 = f.x1; tr.t.y1 = f.y1; tr.t.z1 = f.z1;
    tr.t.x2 = f.x2; tr.t.y2 = f.y2; tr.t.z2 = f.z2;
    e = exit_bit(tr.t);
  }
  advance(tr.ch, tr.t, e);
  return kContinue;
}

// Per-pixel ray direction (cell/ppu_renderer.cpp:56) + AdjustDir (eps 1e-5).
__device__ __forceinline__ void pixel_dir(const SvoFrameArgs& a, int x, int y, float& dx,
                                          float& dy, float& dz) {
  const float fx = (float)x, fy = (float)y;
  dx = __fadd_rn(__fadd_rn(a.dir0[0], __fmul_rn(a.du[0], fx)), __fmul_rn(a.dv[0], fy));
  dy = __fadd_rn(__fadd_rn(a.dir0[1], __fmul_rn(a.du[1], fx)), __fmul_rn(a.dv[1], fy));
  dz = __fadd_rn(__fadd_rn(a.dir0[2], __fmul_rn(a.du[2], fx)), __fmul_rn(a.dv[2], fy));
  const float len = __fsqrt_rn(
      __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
  dx = __fdiv_rn(dx, len);
  dy = __fdiv_rn(dy, len);
  dz = __fdiv_rn(dz, len);
  const float eps = 1e-5f;
  if (fabsf(dx) < eps) dx = copysignf(eps, dx);
  if (fabsf(dy) < eps) dy = copysignf(eps, dy);
  if (fabsf(dz) < eps) dz = copysignf(eps, dz);
}

// Shading record of a leaf: x = RGBA8, y/z/w = the unit normal in FP32
// (int8 normal / its length, each a round-to-nearest operation; zero for a
// zero normal).  The library's layout stores these records (normalised once
// on the host); a caller's 8-byte yv_leaf_attr is normalised here.
__device__ __forceinline__ uint4 shading_record(uint2 at) {
  const float nx = (float)(int8_t)(at.y & 0xFFu);
  const float ny = (float)(int8_t)((at.y >> 8) & 0xFFu);
  const float nz = (float)(int8_t)((at.y >> 16) & 0xFFu);
  const float len2 =
      __fadd_rn(__fadd_rn(__fmul_rn(nx, nx), __fmul_rn(ny, ny)), __fmul_rn(nz, nz));
  float ux = 0.f, uy = 0.f, uz = 0.f;
  if (len2 > 0.f) {
    const float len = __fsqrt_rn(len2);
    ux = __fdiv_rn(nx, len);
    uy = __fdiv_rn(ny, len);
    uz = __fdiv_rn(nz, len);
  }
  return make_uint4(at.x, __float_as_uint(ux), __float_as_uint(uy), __float_as_uint(uz));
}

template <bool kRef>
__device__ __forceinline__ uint4 load_shading(const SvoDeviceScene& sc, uint32_t leaf) {
  if (kRef) return shading_record(__ldg(static_cast<const uint2*>(sc.attrs) + leaf));
  return __ldg(static_cast<const uint4*>(sc.attrs) + leaf);
}

// Hit word of a ray that ended at child tr.ch of tr.node, and its attribute:
// `leaf` as trace_step left it.
template <bool kRef>
__device__ __forceinline__ uint32_t hit_word(const SvoDeviceScene& sc, const Trace& tr,
                                             uint32_t& leaf) {
  const uint32_t c = tr.ch ^ tr.df;  // x 4
  if (kRef) return (tr.node << 3) | (c >> 2);
  const uint2 cold = __ldg(sc.cold + tr.node);
  if (leaf == kLeafOfNode) {
    // leaf codes (both top bits of the nibble) of the children before this one
    const uint32_t before = tr.codes & (tr.codes << 1) & 0x88888888u & ~(0xFFFFFFFFu >> c);
    leaf = cold.y + __popc(before);
    if (sc.leaf_attr) leaf = __ldg(sc.leaf_attr + leaf);
  }
  return (cold.x << 3) | (c >> 2);
}

// Lambert: ambient + diffuse*max(0, n.L) (ambient only in shadow).
__device__ __forceinline__ uint32_t shade(uint4 at, const SvoFrameArgs& a, bool shadowed) {
  const float ndl = __fadd_rn(__fadd_rn(__fmul_rn(__uint_as_float(at.y), a.light[0]),
                                        __fmul_rn(__uint_as_float(at.z), a.light[1])),
                              __fmul_rn(__uint_as_float(at.w), a.light[2]));
  const float dif = ndl > 0.f ? ndl : 0.f;
  const float inten = shadowed ? a.ambient : __fadd_rn(a.ambient, __fmul_rn(a.diffuse, dif));
  uint32_t out = 0xFF000000u;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float v = __fadd_rn(__fmul_rn((float)((at.x >> (8 * c)) & 0xFFu), inten), 0.5f);
    const uint32_t u = v >= 255.f ? 255u : __float2uint_rz(v);
    out |= u << (8 * c);
  }
  return out;
}

// What a pixel's primary ray gives: hit word, t, fetches and the normal of
// the hit leaf's shading record `at` (zero for a miss).
__device__ __forceinline__ void write_primary(const SvoFrameArgs& a, uint32_t off,
                                              uint32_t hitw, float ht, uint32_t f,
                                              uint4 at = make_uint4(0u, 0u, 0u, 0u)) {
  if (a.hit) a.hit[off] = hitw;
  if (a.hit_t) a.hit_t[off] = ht;
  if (a.fetches) a.fetches[off] = f;
  if (a.normal) {
    const size_t n = 3u * (size_t)off;  // off < 2^31: 3 off needs 64 bits
    a.normal[n] = __uint_as_float(at.y);
    a.normal[n + 1u] = __uint_as_float(at.z);
    a.normal[n + 2u] = __uint_as_float(at.w);
  }
}

// What is known once its shadow ray has ended too (or there is none).
__device__ __forceinline__ void write_color(const SvoFrameArgs& a, uint32_t off, uint32_t rgba,
                                            uint32_t fs) {
  if (a.rgba) a.rgba[off] = rgba;
  if (a.shadow_fetches) a.shadow_fetches[off] = fs;
}

__device__ __forceinline__ void write_miss(const SvoFrameArgs& a, uint32_t off, uint32_t f) {
  write_primary(a, off, 0xFFFFFFFFu, 0.f, f);
  write_color(a, off, 0u, 0u);
}

// Origin of the shadow ray of the hit tr ended at: the hit point of the
// primary ray (pos + d t) moved half a leaf out through the entry face.
__device__ __forceinline__ void shadow_origin(const SvoFrameArgs& a, const Trace& tr, float dx,
                                              float dy, float dz, float ht, float* o) {
  o[0] = __fadd_rn(a.pos[0], __fmul_rn(dx, ht));
  o[1] = __fadd_rn(a.pos[1], __fmul_rn(dy, ht));
  o[2] = __fadd_rn(a.pos[2], __fmul_rn(dz, ht));
  int e = 0;
  float m = tr.t.x1;
  if (tr.t.y1 > m) { e = 1; m = tr.t.y1; }
  if (tr.t.z1 > m) e = 2;
  const float half = __int_as_float((127 - (tr.level + 2)) << 23);
  const float d_off = ((tr.df >> (2 + e)) & 1u) ? half : -half;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (e == i) o[i] = __fadd_rn(o[i], d_off);
}

// kMinBlocks: resident 256-thread blocks per SM the register allocation is
// sized for (the occupancy / register-spill trade-off is autotuned).
// kRef: the node pool is the reference VoxNode layout (hit ids are then the
// pool's own node indices); otherwise the library's device layout.
// kRing: frames of the per-lane shared-memory ring (0: local memory only);
// kStaged: the first nsm node records are copied to shared memory and read
// there (measured: reading every record through L1 is as fast or faster,
// so the default is unstaged and nsm = 0).
// Dynamic shared memory = 8 B x nsm staged nodes + 1 KB x kRing per warp.
// kLod: level-of-detail cut-off (a.lod_coef, sc.node_data; library layout).
// kShared: the scene has a table of children.
// lanes: rays a warp takes at a time (the other lanes stay idle), for frames
// too small to fill the GPU (frame_lanes).
template <int kMinBlocks, bool kRef, int kRing, bool kStaged, bool kLod = false,
          bool kShared = false>
__global__ void __launch_bounds__(256, kMinBlocks)
    svo_frame_kernel(SvoDeviceScene sc, SvoFrameArgs a, uint32_t nsm, uint32_t refill_min,
                     uint32_t lanes) {
  extern __shared__ uint4 smem[];
  // the block's deadline under a frame budget (held in shared memory, not
  // in a register of the traversal)
  __shared__ unsigned long long deadline;
  if (!kStaged) nsm = 0;
  nsm &= ~1u;  // whole 16-byte pairs of records
  for (uint32_t i = threadIdx.x; i < nsm / 2; i += blockDim.x)
    smem[i] = __ldg(reinterpret_cast<const uint4*>(sc.nodes) + i);
  if (threadIdx.x == 0 && a.budget_us)
    deadline = global_timer_ns() + 1000ull * (unsigned long long)a.budget_us;
  __syncthreads();
  const uint32_t* smw = reinterpret_cast<const uint32_t*>(smem);
  uint4* ring = smem + nsm / 2 + (threadIdx.x >> 5) * (2 * kRing * 32) + (threadIdx.x & 31u);

  Frame stk[YV_MAX_DEPTH];
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const uint32_t tiles_x = (uint32_t)((a.width + 7) >> 3);
  const uint32_t n_ids = a.id_end;
  uint32_t err = 0, my_hits = 0, my_shadowed = 0;

  uint32_t mode = lane < lanes ? kIdle : kDone, off = 0;
  Trace tr;
  float dx = 0.f, dy = 0.f, dz = 0.f;
  // colours of the pixel whose shadow ray is under way, lit and in shadow
  uint32_t lit = 0, dark = 0;

  for (;;) {
    // ---- refill idle lanes from the global ray counter ----
    const uint32_t idle = __ballot_sync(0xFFFFFFFFu, mode == kIdle);
    // past the frame budget: the idle lanes take no new rays (lane 0's
    // reading of the timer decides for the warp)
    if (idle && a.budget_us &&
        __shfl_sync(0xFFFFFFFFu, global_timer_ns() > deadline ? 1 : 0, 0)) {
      if (mode == kIdle) mode = kDone;
      if (lane == 0) err |= YV_DEV_ERR_TIMEOUT;
    } else if (idle) {
      const uint32_t leader = (uint32_t)__ffs(idle) - 1u;
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(&a.counters[0], (uint32_t)__popc(idle));
      base = __shfl_sync(0xFFFFFFFFu, base, (int)leader);
      if (mode == kIdle) {
        const uint32_t id = a.id_begin + base + (uint32_t)__popc(idle & lt_mask);
        if (id >= n_ids) {
          mode = kDone;
        } else {
          const uint32_t tile = id >> 5, w = id & 31u;
          // a tile's two 4x4 halves, each in rows of 4: any 4, 8 or 16
          // consecutive ids are neighbouring pixels
          const int x = (int)((tile % tiles_x) * 8u + ((w & 3u) | ((w >> 2) & 4u)));
          const int y = (int)((tile / tiles_x) * 4u + ((w >> 2) & 3u));
          if (x < a.width && y < a.height) {
            off = (uint32_t)y * (uint32_t)a.width + (uint32_t)x;
            pixel_dir(a, x, y, dx, dy, dz);
            if (begin_trace<kRef, kStaged>(sc, smw, nsm, a.pos[0], a.pos[1], a.pos[2], dx, dy,
                                           dz, tr, err)) {
              mode = kPrimary;
            } else {
              write_miss(a, off, tr.fetches);
            }
          }
        }
      }
    }
    if (__all_sync(0xFFFFFFFFu, mode == kDone)) break;

    // ---- trace until refill_min lanes (or all) are free: up to kStepsPerVote
    // steps per warp vote, the end of a ray handled once after them (a lane
    // whose ray ended idles for the rest of the group) ----
    for (;;) {
      int r = kContinue;
      uint32_t leaf = 0;
#pragma unroll 6
      for (int k = 0; k < kStepsPerVote; ++k)
        if ((mode == kPrimary || mode == kShadow) && r == kContinue)
          r = trace_step<kRef, kRing, kStaged, kLod, kShared>(
              sc, smw, nsm, stk, ring, tr, mode == kShadow, leaf, err, a.lod_coef);
      if (r != kContinue) {
        if (mode == kShadow) {
          // end of a shadow ray
          const bool sh = r == kHit;
          my_shadowed += sh ? 1u : 0u;
          write_color(a, off, sh ? dark : lit, tr.fetches);
          mode = kIdle;
        } else if (r == kMiss) {
          write_miss(a, off, tr.fetches);
          mode = kIdle;
        } else {
          // everything but the colour is written now: the shadow ray carries
          // two words along instead of the hit and its shading record (46
          // registers at 5 blocks an SM, none spilled: 540 -> 526 us)
          ++my_hits;
          const uint32_t hitw = hit_word<kRef>(sc, tr, leaf);
          const float ht = max3f(tr.t.x1, tr.t.y1, tr.t.z1);
          uint4 attr = make_uint4(0u, 0u, 0u, 0u);
          if (leaf < sc.n_attrs)
            attr = load_shading<kRef>(sc, leaf);
          else
            err |= YV_DEV_ERR_POOL;
          write_primary(a, off, hitw, ht, tr.fetches, attr);
          lit = shade(attr, a, false);
          mode = kIdle;
          if (a.shadows) {
            dark = shade(attr, a, true);
            float o[3];
            shadow_origin(a, tr, dx, dy, dz, ht, o);
            if (begin_trace<kRef, kStaged>(sc, smw, nsm, o[0], o[1], o[2], a.light_ray[0],
                                           a.light_ray[1], a.light_ray[2], tr, err))
              mode = kShadow;
            else
              write_color(a, off, lit, tr.fetches);
          } else {
            write_color(a, off, lit, 0u);
          }
        }
      }
      const uint32_t free_lanes = __ballot_sync(0xFFFFFFFFu, mode == kIdle || mode == kDone);
      if (free_lanes == 0xFFFFFFFFu || __popc(free_lanes) >= (int)refill_min) break;
    }
  }

  // block totals of the counters, one atomic per block and counter
  __shared__ uint32_t red[3];
  if (threadIdx.x < 3) red[threadIdx.x] = 0;
  __syncthreads();
  if (my_hits) atomicAdd(&red[0], my_hits);
  if (my_shadowed) atomicAdd(&red[1], my_shadowed);
  if (err) atomicOr(&red[2], err);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (red[0]) atomicAdd(&a.counters[2], red[0]);
    if (red[1]) atomicAdd(&a.counters[3], red[1]);
    if (red[2]) atomicOr(&a.counters[1], red[2]);
  }
}

}  // namespace
}  // namespace yv
