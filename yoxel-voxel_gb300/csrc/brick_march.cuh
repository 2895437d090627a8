// brick_march.cuh - device code of the brick-volume ray-march (ntree layout)
// for sm_103a, shared by brick_kernels.cu and batch_kernels.cu.
//
// March (restating castRay / walkBrick / intersect of
// reaction/trace/trace.cu:42-139 over the N=4 grid tree of volume_host.cpp):
//  * clip the ray to the unit cube, t_enter = max(t_enter, 0);
//  * DDA over brick cells; cell c spans [t_in, t_out) with t_in = the
//    previous cell's t_out, so cells partition the ray;
//  * in an occupied cell, samples sit at the global multiples t = k*dt
//    (trace.cu:47), dt = step_vox lattice cells;
//  * sample = software FP32 trilinear of density and albedo inside the brick
//    (the 9^3 apron lattice keeps all 8 corners in the brick), at a position
//    carried as a float pair (sample_coords) so the trilinear fractions are
//    accurate to ulp(1);
//  * alpha = saturate(alpha_scale * density), front-to-back pre-multiplied
//    accumulation C += (1-A)*alpha*albedo, A += (1-A)*alpha (trace.cu:58),
//    stop once A > 0.99 (trace.cu:59).
// Every float operation of the march is an explicit round-to-nearest
// intrinsic so the forward and the backward kernels replay bit-identical
// values (the adjoint relies on reaching the forward's exact final colour).
//
// Adjoint: the backward kernel re-marches each ray instead of storing
// per-sample state.  With T = 1 - A before sample j and the forward output
// (C, A) of the ray:
//   d out_k / d alpha_j = T c_jk - (out_k - out_k after j) / (1 - alpha_j)
//   d out_k / d c_jk    = T alpha_j            (c_A = 1)
// Gradients for the 8 trilinear corners are coalesced in registers while
// consecutive samples of a ray stay in the same trilinear cell, then flushed
// with FP32 vector atomics: one of 16 bytes per corner, or per edge of the cell
// in x one of 8 bytes (no colour) or two of 16 (GradVis in brick_kernels.cu).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "yv_volume.h"

namespace yv {
namespace {

constexpr int kL = 9;
constexpr int kL3 = 729;
constexpr uint32_t kEmpty = 0x80000000u;
constexpr uint32_t kBrick = 0x40000000u;

__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float ffma(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// Exact conversions on the ALU / FMA pipes instead of the conversion unit
// (which runs at a fraction of their rate); used where they measured faster
// (the 8-byte packed format).
// Byte k of v as a float: 2^23 + byte assembled by one byte permute, minus
// 2^23 (exact).
__device__ __forceinline__ float byte_f(uint32_t v, int k) {
  return __fsub_rn(__uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440u + (uint32_t)k)),
                   8388608.f);
}
// Pairs of floats in one 64-bit register pair and their packed operations, each
// half rounded as the scalar one: one instruction to issue for two.  The march
// is bound by issue: the corner sums as pairs took 1024^2 of a 512^3 volume
// 695 -> 680 us and a 64-camera fitting step 8.93 -> 8.64 ms, the weights,
// bytes and coordinates as pairs too 667 us and 8.52 ms, a 16-scene batch 2067
// -> 1935 us.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

template <int P>
struct Voxel;

// Lattice formats (VolumeView::precision).  corner() loads one lattice
// point: density and the three albedo channels (raw 0..255 for the uint8
// formats, scaled once after interpolation by kAlbedoScale).
//   0: fp16 density array + uchar4 albedo array (two loads)
//   1: fp32 density array + fp32 RGB albedo array (learnable; four loads)
//   2: packed float4 (r, g, b, density) (one 16-byte load)
//   3: packed 8 bytes {fp16 density | r << 16 | g << 24, b} (one 8-byte load)
template <>
struct Voxel<0> {
  static constexpr float kAlbedoScale = 1.0f / 255.0f;
  __device__ static __forceinline__ void corner(const VolumeView& a, uint32_t i, float& d,
                                                float* c) {
    d = __half2float(__ushort_as_half(__ldg(static_cast<const unsigned short*>(a.density) + i)));
    const uint32_t v = __ldg(static_cast<const unsigned int*>(a.albedo) + i);
    c[0] = (float)(v & 0xFFu);
    c[1] = (float)((v >> 8) & 0xFFu);
    c[2] = (float)((v >> 16) & 0xFFu);
  }
};

template <>
struct Voxel<1> {
  static constexpr float kAlbedoScale = 1.0f;
  __device__ static __forceinline__ void corner(const VolumeView& a, uint32_t i, float& d,
                                                float* c) {
    d = __ldg(static_cast<const float*>(a.density) + i);
    const float* q = static_cast<const float*>(a.albedo) + 3 * (size_t)i;
    c[0] = __ldg(q);
    c[1] = __ldg(q + 1);
    c[2] = __ldg(q + 2);
  }
};

template <>
struct Voxel<2> {
  static constexpr float kAlbedoScale = 1.0f;
  __device__ static __forceinline__ void corner(const VolumeView& a, uint32_t i, float& d,
                                                float* c) {
    const float4 v = __ldg(static_cast<const float4*>(a.albedo) + i);
    c[0] = v.x;
    c[1] = v.y;
    c[2] = v.z;
    d = v.w;
  }
};

template <>
struct Voxel<3> {
  static constexpr float kAlbedoScale = 1.0f / 255.0f;
  __device__ static __forceinline__ void corner(const VolumeView& a, uint32_t i, float& d,
                                                float* c) {
    const uint2 v = __ldg(static_cast<const uint2*>(a.albedo) + i);
    d = __half2float(__ushort_as_half((unsigned short)(v.x & 0xFFFFu)));
    const float m = -8388608.f;
    unpack2(add2(pack2(__uint_as_float(__byte_perm(v.x, 0x4B000000u, 0x7442u)),
                       __uint_as_float(__byte_perm(v.x, 0x4B000000u, 0x7443u))),
                 pack2(m, m)),
            c[0], c[1]);
    c[2] = byte_f(v.y, 0);
  }
};

struct SampleCtx {
  uint32_t base;  // brick*729 + corner-000 lattice index
  float w[8];     // trilinear weights, corner j: bit0 +x, bit1 +y, bit2 +z
  float sigma, alpha;
  float col[3];
};

// Lattice offset of trilinear corner j inside a 9^3 brick.
__device__ __forceinline__ uint32_t corner_offset(int j) {
  return (uint32_t)(((j >> 2) * kL + ((j >> 1) & 1)) * kL + (j & 1));
}

// a + b as an exact float pair s + r (Knuth's TwoSum).
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& r) {
  s = fadd(a, b);
  const float bb = fsub(s, a);
  r = fadd(fsub(a, fsub(s, bb)), fsub(b, bb));
}

// Brick-local lattice coordinate t D + (Lh + Ll) of a sample (in [0, 8]),
// Lh + Ll the brick-local origin o S - 8c as an exact pair (two_sum: o S is
// exact, but o S - 8c can need one bit more when it grows a binade), as a
// float pair l + e: p = t D rounded, e = its exact rounding error (one fma)
// plus Ll, l = p + Lh.  Once the origin is more than two bricks away, p and
// -Lh agree to a factor of two and l is exact (Sterbenz), so the fractional
// position inside the trilinear cell, (l - k) + e, is accurate to ulp(1)
// instead of ulp(8) or ulp(o S).  (Rounded once to ulp(8), and o S - 8c to
// ulp(o S), sample points on steep density edges moved low-opacity rays by
// up to 5e-5 relative.)
__device__ __forceinline__ void sample_coords(float t, const float* D, const float* Lh,
                                              const float* Ll, float* l, float* e) {
  const f32x2 t2 = pack2(t, t), D2 = pack2(D[0], D[1]), p2 = mul2(t2, D2);
  float p0, p1;
  unpack2(p2, p0, p1);
  unpack2(add2(fma2(t2, D2, pack2(-p0, -p1)), pack2(Ll[0], Ll[1])), e[0], e[1]);
  unpack2(add2(p2, pack2(Lh[0], Lh[1])), l[0], l[1]);
  const float p = fmul(t, D[2]);
  e[2] = fadd(ffma(t, D[2], -p), Ll[2]);
  l[2] = fadd(p, Lh[2]);
}

// floor of a lattice coordinate clamped to cell 0..7 as 2^23 + k, the integer
// k in its low bits (0x4B000000 | k): one add that rounds down, in place of a
// conversion (quarter rate) and integer clamps.
__device__ __forceinline__ float cell_of(float l) {
  return __fadd_rd(fminf(fmaxf(l, 0.f), 7.f), 8388608.f);
}

// Whether the cell kb (cell_of) of brick b has its bit in the cell occupancy
// mask: bit (y & 3) * 8 + x of word z * 2 + (y >> 2).  The constants that
// cell_of adds vanish in the shift (modulo 32) and cancel in the word index.
__device__ __forceinline__ bool cell_marked(const VolumeView& a, int b, const float* kb) {
  const uint32_t x = __float_as_uint(kb[0]), y = __float_as_uint(kb[1]),
                 z = __float_as_uint(kb[2]);
  const uint32_t w = (uint32_t)b * 16u - 0x4B000000u * 2u - (0x4B000000u >> 2) + z * 2u + (y >> 2);
  return (__ldg(a.cell_mask + w) >> ((y * 8u + x) & 31u)) & 1u;
}

// l + e: brick-local lattice coordinates of the sample (sample_coords), in
// [0, 8]; kb its cell (cell_of).
template <int P>
__device__ __forceinline__ void eval_sample(const VolumeView& a, int b, const float* l,
                                            const float* e, const float* kb, SampleCtx& s) {
  float f[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    // saturate: a fraction a rounding outside [0, 1] is clamped
    f[i] = __saturatef(fadd(fsub(l[i], fsub(kb[i], 8388608.f)), e[i]));
  }
  // k + 0x4B000000 in each coordinate: the constants cancel modulo 2^32
  s.base = (uint32_t)b * (uint32_t)kL3 - 0x4B000000u * 91u + __float_as_uint(kb[2]) * 81u +
           __float_as_uint(kb[1]) * 9u + __float_as_uint(kb[0]);
  const float gx = fsub(1.f, f[0]), gy = fsub(1.f, f[1]), gz = fsub(1.f, f[2]);
  const f32x2 x2 = pack2(gx, f[0]);
  const f32x2 y0 = mul2(x2, pack2(gy, gy)), y1 = mul2(x2, pack2(f[1], f[1]));
  const f32x2 z0 = pack2(gz, gz), z1 = pack2(f[2], f[2]);
  unpack2(mul2(y0, z0), s.w[0], s.w[1]);
  unpack2(mul2(y1, z0), s.w[2], s.w[3]);
  unpack2(mul2(y0, z1), s.w[4], s.w[5]);
  unpack2(mul2(y1, z1), s.w[6], s.w[7]);
  f32x2 rg = 0ull, bd = 0ull;  // (r, g) and (b, density) of the sample
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float dj, c[3];
    Voxel<P>::corner(a, s.base + corner_offset(j), dj, c);
    const f32x2 w = pack2(s.w[j], s.w[j]);
    rg = fma2(w, pack2(c[0], c[1]), rg);
    bd = fma2(w, pack2(c[2], dj), bd);
  }
  float sig, c0, c1, c2;
  unpack2(rg, c0, c1);
  unpack2(bd, c2, sig);
  s.sigma = sig;
  s.col[0] = fmul(c0, Voxel<P>::kAlbedoScale);
  s.col[1] = fmul(c1, Voxel<P>::kAlbedoScale);
  s.col[2] = fmul(c2, Voxel<P>::kAlbedoScale);
  float al = fmul(s.sigma, a.alpha_scale);
  s.alpha = al < 0.f ? 0.f : (al > 1.f ? 1.f : al);
}

// Tree descent for brick cell `cell` (ntree/ntree/nodes.h:56-99 offsets).
// Every node is read through L1.  Returns brick id, -1 if empty, -2 if the
// pool is malformed.
__device__ __forceinline__ int lookup(const VolumeView& a, const int* cell) {
  uint32_t node = 0;
  for (int lev = 0; lev < a.levels; ++lev) {
    const int sh = 2 * (a.levels - 1 - lev);
    const uint32_t c = (uint32_t)((((cell[2] >> sh) & 3) * 4 + ((cell[1] >> sh) & 3)) * 4 +
                                  ((cell[0] >> sh) & 3));
    if (node >= a.ngrids) return -2;
    const uint32_t ref = __ldg(a.grids + (size_t)node * 64 + c);
    if (ref & kEmpty) return -1;
    if (ref & kBrick) {
      const uint32_t b = ref & 0x3FFFFFFFu;
      return (lev == a.levels - 1 && b < a.nbricks) ? (int)b : -2;
    }
    if (lev == a.levels - 1) return -2;
    node = ref;
  }
  return -1;
}

struct RayOut {
  float c[3];
  float a;
  uint32_t samples;
  uint32_t bricks;
  bool bad;
};

// State of one ray's march: the DDA over brick cells and, inside an occupied
// one, the run of its samples.
// kLean keeps less of it alive for the adjoint's tighter register budget: the
// step direction of an axis is the sign of inv (d is never 0), and the
// lattice-space origin o S is recomputed (the same rounded product) at each
// occupied cell.
template <bool kLean>
struct March {
  float inv[3], D[3], Q[kLean ? 1 : 3];  // 1 / d; lattice-space direction, origin
  int cell[3];
  float t_in, t_out;
  int e;  // exit axis of the current cell
  // occupied cell: brick, its local origin as an exact pair, next sample
  int b, k;
  float Lh[3], Ll[3], t;
};

// Clips the ray to the unit cube; false: it misses.
template <bool kLean>
__device__ __forceinline__ bool march_begin(const VolumeView& a, const float* o, const float* d,
                                            March<kLean>& m) {
  float t1[3], t2[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    m.inv[i] = __fdiv_rn(1.f, d[i]);
    const float lo = fmul(fsub(0.f, o[i]), m.inv[i]);
    const float hi = fmul(fsub(1.f, o[i]), m.inv[i]);
    t1[i] = lo < hi ? lo : hi;
    t2[i] = lo < hi ? hi : lo;
  }
  float t_enter = fmaxf(fmaxf(t1[0], t1[1]), t1[2]);
  const float t_exit = fminf(fminf(t2[0], t2[1]), t2[2]);
  if (t_enter < 0.f) t_enter = 0.f;
  if (t_exit < 0.f || t_enter > t_exit) return false;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float q = __fdiv_rn(fadd(o[i], fmul(t_enter, d[i])), a.cell_size);
    int k = __float2int_rd(q);
    m.cell[i] = k < 0 ? 0 : (k > a.nb - 1 ? a.nb - 1 : k);
    if (!kLean) m.Q[i] = fmul(o[i], a.S);
    m.D[i] = fmul(d[i], a.S);
  }
  m.t_in = t_enter;
  return true;
}

// The current brick cell: its exit and what the tree holds there (brick id,
// -1 empty, -2 malformed).
template <bool kLean>
__device__ __forceinline__ int march_cell(const VolumeView& a, const float* o, March<kLean>& m) {
  float tx[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const bool up = m.inv[i] > 0.f;
    const float plane = fmul((float)(up ? m.cell[i] + 1 : m.cell[i]), a.cell_size);
    tx[i] = fmul(fsub(plane, o[i]), m.inv[i]);
  }
  // exit axis = first argmin (selects, no dynamic register indexing)
  m.e = 0;
  m.t_out = tx[0];
  if (tx[1] < m.t_out) { m.e = 1; m.t_out = tx[1]; }
  if (tx[2] < m.t_out) { m.e = 2; m.t_out = tx[2]; }
  // the tree is descended only where the brick bitmap (if any) says a brick
  // may be
  const uint32_t ci =
      ((uint32_t)m.cell[2] * (uint32_t)a.nb + (uint32_t)m.cell[1]) * (uint32_t)a.nb +
      (uint32_t)m.cell[0];
  if (a.brick_bits && !((__ldg(a.brick_bits + (ci >> 5)) >> (ci & 31u)) & 1u)) return -1;
  return lookup(a, m.cell);
}

// Into the next brick cell; false: the ray leaves the volume.
template <bool kLean>
__device__ __forceinline__ bool march_next(const VolumeView& a, March<kLean>& m) {
  m.t_in = m.t_out;
  int ce;
  if (m.e == 0) ce = (m.cell[0] += m.inv[0] > 0.f ? 1 : -1);
  else if (m.e == 1) ce = (m.cell[1] += m.inv[1] > 0.f ? 1 : -1);
  else ce = (m.cell[2] += m.inv[2] > 0.f ? 1 : -1);
  return ce >= 0 && ce < a.nb;
}

// The samples of the occupied cell b: the brick-local origin Q - 8c as an
// exact pair - the brick-local coordinate t D + (Q - 8c) in [0, 8] is formed
// without the rounding of |Q| (sample_coords) - and the first sample.
template <bool kLean>
__device__ __forceinline__ void march_enter(const VolumeView& a, const float* o, int b,
                                            March<kLean>& m) {
  m.b = b;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    two_sum(kLean ? fmul(o[i], a.S) : m.Q[kLean ? 0 : i], -(float)(8 * m.cell[i]), m.Lh[i],
            m.Ll[i]);
  m.k = __float2int_ru(fmul(m.t_in, a.inv_dt));
  m.t = fmul((float)m.k, a.dt);
}

// One ray; `Vis` is called per sample with (sample, T, T alpha).
// kColor = false (the adjoint's replay): the composited colour is not
// accumulated (the visitor tracks what it needs; r.c stays 0).
// kSkip: the forward passes over the samples of cells the pool's
// cell_mask marks empty where `masked` (compiled out for pools without one).
template <int P, class Vis, bool kColor = true, bool kSkip = kColor>
__device__ __forceinline__ void march(const VolumeView& a, const float* o, const float* d,
                                      Vis& vis, RayOut& r, bool masked = false) {
  r.c[0] = r.c[1] = r.c[2] = 0.f;
  r.a = 0.f;
  r.samples = 0;
  r.bricks = 0;
  r.bad = false;
  March<!kColor> m;
  if (!march_begin(a, o, d, m)) return;
  float A = 0.f, C0 = 0.f, C1 = 0.f, C2 = 0.f;
  for (int guard = 0; guard < 4 * 4096; ++guard) {
    const int b = march_cell(a, o, m);
    if (b == -2) {
      r.bad = true;
      break;
    }
    if (b >= 0) {
      ++r.bricks;
      march_enter(a, o, b, m);
      for (int it = 0; it < 1 << 16; ++it, ++m.k, m.t = fmul((float)m.k, a.dt)) {
        if (!(m.t < m.t_out)) break;
        float lc[3], le[3], kb[3];
        sample_coords(m.t, m.D, m.Lh, m.Ll, lc, le);
#pragma unroll
        for (int i = 0; i < 3; ++i) kb[i] = cell_of(lc[i]);
        if (kColor && kSkip && masked && !cell_marked(a, b, kb)) {
          // a cell whose 8 corners are all zero has sigma = 0, alpha = 0:
          // the sample adds exactly nothing (C, A unchanged), so the
          // forward passes over it; the replay of the adjoint, whose
          // density gradient reaches such samples, takes every sample
          ++r.samples;
          continue;
        }
        SampleCtx s;
        eval_sample<P>(a, b, lc, le, kb, s);
        const float T = fsub(1.f, A);
        const float w = fmul(T, s.alpha);
        vis(s, T, w);
        if (kColor) {
          C0 = ffma(w, s.col[0], C0);
          C1 = ffma(w, s.col[1], C1);
          C2 = ffma(w, s.col[2], C2);
        }
        A = fadd(A, w);
        ++r.samples;
        if (A > 0.99f) goto done;
      }
    }
    if (!march_next(a, m)) break;
  }
done:
  r.c[0] = C0;
  r.c[1] = C1;
  r.c[2] = C2;
  r.a = A;
}

struct NoVis {
  __device__ __forceinline__ void operator()(const SampleCtx&, float, float) {}
};

__device__ __forceinline__ void pixel_ray(const CamBasis& c, int x, int y, float* o, float* d) {
  const float fx = (float)x, fy = (float)y;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    o[i] = c.pos[i];
    d[i] = fadd(fadd(c.dir0[i], fmul(c.du[i], fx)), fmul(c.dv[i], fy));
  }
  const float len = __fsqrt_rn(fadd(fadd(fmul(d[0], d[0]), fmul(d[1], d[1])), fmul(d[2], d[2])));
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    d[i] = __fdiv_rn(d[i], len);
    if (fabsf(d[i]) < 1e-5f) d[i] = copysignf(1e-5f, d[i]);
  }
}

}  // namespace
}  // namespace yv
