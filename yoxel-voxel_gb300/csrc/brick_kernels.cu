// brick_kernels.cu - brick-volume ray-march kernels (ntree layout) for
// sm_103a: forward compositing over many cameras, the re-marching adjoint,
// and apron maintenance.  Device helpers and the march are in
// brick_march.cuh.
#include "brick_march.cuh"
#include "brick_mask.cuh"

#include <atomic>

namespace yv {
namespace {

// Threads of a march block: half of a 16x16-pixel square.  A block holds its
// registers until its slowest warp ends, so smaller blocks keep more warps at
// work: 64-camera training step 10.04 ms at 256 threads, 9.66 at 128, 9.79 at
// 64; 1024^2 frame of a 512^3 volume 740 / 704 / 719 us.
constexpr int kMarchThreads = 128;
// Register budgets (resident warps per SM / 8).  A launch that fills the GPU
// runs at 3: adjoint of a 64-camera fitting step of a 128^3 volume 6.5 ms (2:
// 6.9, 4: 6.9 with spills); forward of the fp32 formats alike at 3 and 4 there
// and 7 % faster at 3 on a volume without empty cells; 8-byte format 1024^2
// of a 512^3 volume 740 us at 3, 764 at 4.  A launch whose warps all fit at 2
// is bound by the latency of its longest warp and runs there, where nothing
// spills and more loads are in flight: 4 cameras at 64x64, forward and
// backward, 693 -> 493 us.
constexpr int kMinBlocks = 3;
constexpr int kSmallMinBlocks = 2;

// tile mapping: warp w of the grid -> 8x4 pixel tile of one camera image;
// 8 consecutive tiles are a 2x4-tile (16x16-pixel) square
__host__ __device__ __forceinline__ uint32_t tile_ids(const VolumeArgs& a) {
  const uint32_t tx = (uint32_t)((a.width + 7) >> 3), ty = (uint32_t)((a.height + 3) >> 2);
  return (uint32_t)a.ncams * ((tx + 1) >> 1) * ((ty + 3) >> 2) * 8u;
}
// `sub`: part sub % (32 / a.lanes) of tile sub / (32 / a.lanes), a.lanes rays
// of the tile's two 4x4 halves (each in rows of 4), one per lane from lane 0.
__device__ __forceinline__ bool ray_of_thread(const VolumeArgs& a, uint32_t sub, int& cam, int& x,
                                              int& y) {
  const uint32_t tx = (uint32_t)((a.width + 7) >> 3), ty = (uint32_t)((a.height + 3) >> 2);
  const uint32_t stx = (tx + 1) >> 1, sty = (ty + 3) >> 2;
  const uint32_t per_cam = stx * sty * 8u;
  const uint32_t nsub = 32u / a.lanes, tile = sub / nsub;
  cam = (int)(tile / per_cam);
  const uint32_t r = tile % per_cam, st = r >> 3, w = r & 7u;
  const uint32_t lane = threadIdx.x & 31u, p = (sub % nsub) * a.lanes + lane;
  if (lane >= a.lanes) return false;
  x = (int)(((st % stx) * 2u + (w & 1u)) * 8u + ((p & 3u) | ((p >> 2) & 4u)));
  y = (int)(((st / stx) * 4u + (w >> 1)) * 4u + ((p >> 2) & 3u));
  return cam < a.ncams && x < a.width && y < a.height;
}

// RGBA8 pixel of a composited colour: each channel saturate(v) * 255
// truncated, R in the low byte (float2uint of reaction/trace/utils.h:37-44,
// the uchar4 image of RunTrace, ntree/ntree_trace.cuh:27).
__device__ __forceinline__ uint32_t rgba8_of(float r, float g, float b, float al) {
  const float v[4] = {r, g, b, al};
  uint32_t out = 0;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const float x = v[c] < 0.f ? 0.f : (v[c] > 1.f ? 1.f : v[c]);
    out |= __float2uint_rz(__fmul_rn(x, 255.f)) << (8 * c);
  }
  return out;
}

// Whether to test the cell mask: always where its fill is not known (a.marked
// null), else where less than 45 % of the cells of 32 bricks spread over the
// pool are marked - a test costs about a fifth of a sample.  Forward of a
// fitting step of a 128^3 volume, 16 cameras at 256^2, with / without the
// mask: 37 % marked 1.02 / 1.33 ms, 60 % 1.39 / 1.31 ms, 88 % 1.05 / 0.95 ms.
// The whole warp calls it; the answer changes the time only.
__device__ __forceinline__ bool mask_pays(const VolumeArgs& a) {
  if (!a.marked) return true;
  const uint32_t b = (uint32_t)(((uint64_t)(threadIdx.x & 31u) * a.v.nbricks) >> 5);
  return __reduce_add_sync(0xFFFFFFFFu, __ldg(a.marked + b)) < 32u * 512u * 45u / 100u;
}

// kBlocks: resident warps per SM / 8 the register allocation is sized for.
// Bound by instruction issue.  On the 1024^2 frame of a 512^3 volume (8-byte
// format) 876 -> 740 us from the cell found by one round-down add instead of
// a conversion and clamps, the fraction clamped by the add's saturation, and
// the half decoded by one conversion; 704 us with blocks of 128 threads.
// kSkip: the pool carries a cell occupancy mask (library-owned pools, and a
// learnable pool that the fitting step's forward packs).
template <int P, int kBlocks, bool kSkip>
__global__ void __launch_bounds__(kMarchThreads, 2 * kBlocks) volume_forward_kernel(VolumeArgs a) {
  // the launch's tiles (a range of them for a frame split across GPUs)
  const uint32_t nsub = 32u / a.lanes;
  const uint32_t n_subs = (a.tile_end ? a.tile_end : tile_ids(a)) * nsub;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const bool masked = kSkip && mask_pays(a);
  bool bad = false;
  for (uint32_t sub = a.tile_begin * nsub + blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
       sub < n_subs; sub += warps) {
    int cam, x, y;
    if (!ray_of_thread(a, sub, cam, x, y)) continue;
    float o[3], d[3];
    pixel_ray(a.cam[cam], x, y, o, d);
    NoVis nv;
    RayOut r;
    march<P, NoVis, true, kSkip>(a.v, o, d, nv, r, masked);
    bad |= r.bad;
    const size_t off = ((size_t)cam * a.height + (size_t)y) * a.width + (size_t)x;
    if (a.rgba) reinterpret_cast<float4*>(a.rgba)[off] = make_float4(r.c[0], r.c[1], r.c[2], r.a);
    if (a.rgba8) a.rgba8[off] = rgba8_of(r.c[0], r.c[1], r.c[2], r.a);
    if (a.samples) a.samples[off] = r.samples;
    if (a.bricks_entered) a.bricks_entered[off] = r.bricks;
  }
  if (bad && a.status) atomicOr(a.status, 4u);
}

// Gradient of one sample w.r.t. its alpha (see the header), contracted with
// dL/d(rgba) = g of the ray up front:
//   sum_k g_k d out_k / d alpha = T (g.c) - (g.out - g.C_after) / (1 - alpha)
// with c_A = 1, C_after = C_before + T alpha c, g.out a per-ray constant
// (gout) and gb = g.C_before tracked along the ray (so the replay need not
// composite the colour).  Returns d(sigma) through saturate.  The colour
// gradient of the sample is g_k T alpha: g is constant along the ray, so
// only T alpha needs accumulating per corner.
__device__ __forceinline__ float sample_dsigma(const VolumeArgs* a, float gc, float gout,
                                               float gb, const SampleCtx& s, float T,
                                               float w) {
  const float ga = ffma(w, gc, gb);
  const float om = fsub(1.f, s.alpha);
  // the gradient bar is 1e-4 relative: the hardware reciprocal suffices
  const float inv_om = om > 0.f ? __fdividef(1.f, om) : 0.f;
  const float dal = ffma(T, gc, -fmul(fsub(gout, ga), inv_om));
  const float sa = fmul(s.sigma, a->v.alpha_scale);
  // saturate'(s) = 1 on [0, 1): right derivative at 0 so that empty lattice
  // points still receive gradient
  return (sa >= 0.f && sa < 1.f) ? fmul(dal, a->v.alpha_scale) : 0.f;
}

// Per-lane coalescing of corner gradients while consecutive samples share
// a trilinear cell: per corner, sum w_j dsigma (density) and sum w_j T alpha
// (colour, scaled by g at the flush).  The first sample of a cell sets the
// accumulators.  (Carrying the 4 shared corners over a face-adjacent move
// halves the atomics but measured 1.3x slower: the per-axis cases diverge
// within a warp.)
//
// Flush: an atomic costs by the request, not by the byte.  With kEdges the
// gradient scratch holds 8 floats per lattice point p for the edge (p, p + 1 in
// x):
//   {density p, density p + 1, r p, g p, b p, r p + 1, g p + 1, b p + 1}
// One 8-byte atomic per edge carries the densities of both its ends: 4 for a
// cell that the ray crossed at alpha 0 (most cells), 8 of 16 bytes for one
// with colour.  Without, 4 floats (albedo rgb, density) per point and 8 atomics
// of 16 bytes for either.  64-camera fitting step of a 128^3 volume 8.46 -> 7.51
// ms with edges; a launch that does not fill the GPU is bound by its longest
// warp, not by atomics, and keeps the smaller scratch (4 cameras at 64x64: 494
// us, 542 with edges), as do others where edges don't pay (backward_uses_edges).
template <bool kEdges>
struct GradVis {
  const VolumeArgs* a;
  float g[4];   // dL/d(r,g,b,a) of this ray
  float gout;   // g . (forward output of this ray)
  float gb;     // g . (r, g, b, A) composited before the current sample
  uint32_t base;
  float wsum;    // sum of T alpha over the cell's samples; NaN where g is not
                 // finite (0 x g is not 0 then)
  f32x2 acc[8];  // (density, colour weight)
  __device__ __forceinline__ void init() {
    base = 0xFFFFFFFFu;
    gb = 0.f;
  }
  __device__ __forceinline__ void flush() {
    if (base == 0xFFFFFFFFu) return;
    if (!kEdges) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float d, w;
        unpack2(acc[j], d, w);
        atomicAdd(a->grad_scratch + base + corner_offset(j),
                  make_float4(fmul(g[0], w), fmul(g[1], w), fmul(g[2], w), d));
      }
      return;
    }
    float4* p = a->grad_scratch + 2 * (size_t)base;
    if (wsum == 0.f) {
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        float d0, d1, w;
        unpack2(acc[j], d0, w);
        unpack2(acc[j + 1], d1, w);
        atomicAdd(reinterpret_cast<float2*>(p + 2u * corner_offset(j)), make_float2(d0, d1));
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        float d0, d1, w0, w1;
        unpack2(acc[j], d0, w0);
        unpack2(acc[j + 1], d1, w1);
        atomicAdd(p + 2u * corner_offset(j), make_float4(d0, d1, fmul(g[0], w0), fmul(g[1], w0)));
        atomicAdd(p + 2u * corner_offset(j) + 1,
                  make_float4(fmul(g[2], w0), fmul(g[0], w1), fmul(g[1], w1), fmul(g[2], w1)));
      }
    }
  }
  __device__ __forceinline__ void operator()(const SampleCtx& s, float T, float w) {
    const float gc = ffma(g[2], s.col[2], ffma(g[1], s.col[1], ffma(g[0], s.col[0], g[3])));
    const float ds = sample_dsigma(a, gc, gout, gb, s, T, w);
    gb = ffma(w, gc, gb);
    const f32x2 v = pack2(ds, w);
    if (s.base != base) {
      flush();
      base = s.base;
      if (kEdges) wsum = ffma(0.f, fadd(fadd(g[0], g[1]), g[2]), w);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = mul2(pack2(s.w[j], s.w[j]), v);
    } else {
      if (kEdges) wsum = fadd(wsum, w);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = fma2(pack2(s.w[j], s.w[j]), v, acc[j]);
    }
  }
};

// Gradient (albedo rgb, density) of a lattice point, x its place in its row:
// with kEdges what its own edge and the edge before it hold for it.
template <bool kEdges>
__device__ __forceinline__ float4 point_grad(const float4* __restrict__ p, size_t point, int x) {
  if (!kEdges) return __ldg(p + point);
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (x < 8) {
    const float4 a = __ldg(p + 2 * point), b = __ldg(p + 2 * point + 1);
    v = make_float4(a.z, a.w, b.x, a.x);
  }
  if (x > 0) {
    const float4 a = __ldg(p + 2 * point - 2), b = __ldg(p + 2 * point - 1);
    v.x += b.y;
    v.y += b.z;
    v.z += b.w;
    v.w += a.y;
  }
  return v;
}

// kBlocks: resident warps per SM / 8 the register allocation is sized for.
template <int P, int kBlocks, bool kEdges>
__global__ void __launch_bounds__(kMarchThreads, 2 * kBlocks) volume_backward_kernel(VolumeArgs a) {
  const uint32_t n_subs = tile_ids(a) * (32u / a.lanes);
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  bool bad = false;
  for (uint32_t sub = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); sub < n_subs;
       sub += warps) {
    int cam, x, y;
    if (!ray_of_thread(a, sub, cam, x, y)) continue;
    const size_t off = ((size_t)cam * a.height + (size_t)y) * a.width + (size_t)x;
    const float4 g4 = reinterpret_cast<const float4*>(a.grad_rgba)[off];
    if (g4.x == 0.f && g4.y == 0.f && g4.z == 0.f && g4.w == 0.f) continue;
    const float4 o4 = reinterpret_cast<const float4*>(a.rgba_fwd)[off];
    float o[3], d[3];
    pixel_ray(a.cam[cam], x, y, o, d);
    GradVis<kEdges> gv;
    gv.a = &a;
    gv.g[0] = g4.x; gv.g[1] = g4.y; gv.g[2] = g4.z; gv.g[3] = g4.w;
    gv.gout = ffma(g4.w, o4.w, ffma(g4.z, o4.z, ffma(g4.y, o4.y, fmul(g4.x, o4.x))));
    gv.init();
    RayOut r;
    march<P, GradVis<kEdges>, false>(a.v, o, d, gv, r);
    gv.flush();
    bad |= r.bad;
  }
  if (bad && a.status) atomicOr(a.status, 4u);
}

// Cell occupancy mask: one warp per mask word - the 32 cells (x, y) of four
// rows of one z layer of a brick - sets the bit of every cell with a
// non-zero density corner, as the march reads the corners (format P).
template <int P>
__global__ void cell_mask_kernel(VolumeView v, uint32_t* mask) {
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (warp >= v.nbricks * 16u) return;  // uniform across the warp
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t b = warp >> 4, word = warp & 15u;
  const uint32_t z = word >> 1, y = (word & 1u) * 4u + (lane >> 3), x = lane & 7u;
  const uint32_t base = b * (uint32_t)kL3 + (z * kL + y) * kL + x;
  bool any = false;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float d, c[3];
    Voxel<P>::corner(v, base + corner_offset(j), d, c);
    any |= d != 0.f;
  }
  const uint32_t bits = __ballot_sync(0xFFFFFFFFu, any);
  if (lane == 0) mask[warp] = bits;
}

// Brick bitmap: one warp per word of 32 brick cells, a lane per cell, its
// bit set unless the tree descent finds the cell empty (a malformed ref
// keeps its bit, so the march's own descent still reports it).
__global__ void brick_bits_kernel(VolumeView v, uint32_t* bits, uint32_t nwords) {
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= nwords) return;  // uniform across the warp
  const uint32_t nb = (uint32_t)v.nb, n = nb * nb * nb;
  const uint32_t ci = w * 32u + (threadIdx.x & 31u);
  bool set = false;
  if (ci < n) {
    const int cell[3] = {(int)(ci % nb), (int)((ci / nb) % nb), (int)(ci / (nb * nb))};
    set = lookup(v, cell) != -1;
  }
  const uint32_t word = __ballot_sync(0xFFFFFFFFu, set);
  if ((threadIdx.x & 31u) == 0) bits[w] = word;
}

// Apron fold, pass 1: every owned lattice point (x,y,z < 8) adds the
// gradient its copies received in the aprons of the lower neighbours.
__global__ void fold_gather_kernel(VolumeArgs a, int channels, float* g) {
  const uint32_t n = a.v.nbricks * 512u;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t b = i >> 9, p = i & 511u;
    const int x = (int)(p & 7u), y = (int)((p >> 3) & 7u), z = (int)(p >> 6);
    const uint32_t own = b * kL3 + (uint32_t)((z * kL + y) * kL + x);
    for (int ch = 0; ch < channels; ++ch) {
      float s = g[(size_t)own * channels + ch];
      for (int m = 1; m < 8; ++m) {
        const int dx = m & 1, dy = (m >> 1) & 1, dz = m >> 2;
        if ((dx && x) || (dy && y) || (dz && z)) continue;
        const int nb = a.nbr_dn[(size_t)b * 7 + (m - 1)];
        if (nb < 0) continue;
        const uint32_t cp = (uint32_t)nb * kL3 +
                            (uint32_t)(((z + 8 * dz) * kL + (y + 8 * dy)) * kL + (x + 8 * dx));
        s += g[(size_t)cp * channels + ch];
      }
      g[(size_t)own * channels + ch] = s;
    }
  }
}

// Apron fold, pass 2 (also the apron sync of parameters): every apron slot
// takes the value of the lattice point's owner, or 0 if the owner is absent.
__global__ void fold_scatter_kernel(VolumeArgs a, int channels, float* g) {
  const uint32_t n = a.v.nbricks * (uint32_t)kL3;
  for (uint64_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const uint32_t i = (uint32_t)k;  // (k: n may be within a stride of 2^32)
    const uint32_t b = i / kL3, p = i % kL3;
    const int x = (int)(p % kL), y = (int)((p / kL) % kL), z = (int)(p / (kL * kL));
    const int dx = x == 8, dy = y == 8, dz = z == 8;
    const int m = dx | (dy << 1) | (dz << 2);
    if (!m) continue;
    const int own = a.nbr_up[(size_t)b * 7 + (m - 1)];
    const uint32_t src = (uint32_t)own * kL3 +
                         (uint32_t)(((z - 8 * dz) * kL + (y - 8 * dy)) * kL + (x - 8 * dx));
    for (int ch = 0; ch < channels; ++ch)
      g[(size_t)i * channels + ch] = own >= 0 ? g[(size_t)src * channels + ch] : 0.f;
  }
}

// The march reads the lattice and the grid nodes through L1, and the
// kernels use no shared memory, so they ask for the largest L1 (carveout 0).
// Measured against staging the root and level-1 grid nodes (16.6 KB a
// block) under the driver's default carveout: 64-camera 128^3 forward
// 1365 -> 1434 Mrays/s and adjoint 6.65 -> 6.40 ms; 512^3 fp16 + RGB8
// frame 875 -> 907 Mrays/s (the lowest carveout that still held the staged
// nodes gave half of these gains).
template <void (*kKernel)(VolumeArgs)>
void launch_march(const VolumeArgs& a, uint32_t blocks, cudaStream_t s) {
  static std::atomic<bool> done[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !done[dev].load(std::memory_order_relaxed)) {
    // a hint: a refusal keeps the default configuration and is not reported
    // as the launch's error
    if (cudaFuncSetAttribute(kKernel, cudaFuncAttributePreferredSharedMemoryCarveout, 0) !=
        cudaSuccess)
      cudaGetLastError();
    done[dev].store(true, std::memory_order_relaxed);
  }
  kKernel<<<blocks, kMarchThreads, 0, s>>>(a);
}

// Whether every warp of a march is resident at the small budget.
bool fits_small(uint32_t blocks) {
  return blocks <= (uint32_t)device_sm_count_vol() * 2u * (uint32_t)kSmallMinBlocks;
}

template <int P, bool kSkip>
void launch_forward(const VolumeArgs& a, uint32_t blocks, cudaStream_t s) {
  if (fits_small(blocks))
    launch_march<volume_forward_kernel<P, kSmallMinBlocks, kSkip>>(a, blocks, s);
  else
    launch_march<volume_forward_kernel<P, kMinBlocks, kSkip>>(a, blocks, s);
}

template <int P>
void launch_forward(const VolumeArgs& a, bool skip, uint32_t blocks, cudaStream_t s) {
  if (skip)
    launch_forward<P, true>(a, blocks, s);
  else
    launch_forward<P, false>(a, blocks, s);
}

template <int P, bool kEdges>
void launch_backward(const VolumeArgs& a, uint32_t blocks, cudaStream_t s) {
  if (fits_small(blocks))
    launch_march<volume_backward_kernel<P, kSmallMinBlocks, kEdges>>(a, blocks, s);
  else
    launch_march<volume_backward_kernel<P, kMinBlocks, kEdges>>(a, blocks, s);
}

}  // namespace

uint32_t volume_tiles_per_camera(int width, int height) {
  const uint32_t tx = (uint32_t)((width + 7) >> 3), ty = (uint32_t)((height + 3) >> 2);
  return ((tx + 1) >> 1) * ((ty + 3) >> 2) * 8u;
}

// Rays a warp marches (a.lanes): 32, or 16 or 8 while the launch's rays so
// split still fit the resident warps.  A warp runs every cell and sample that
// any of its rays takes, so a launch too small to fill the GPU ends sooner
// with fewer rays to a warp (4 cameras at 64x64, 128^3 volume, forward and
// backward: 1518 us at 32 rays, 1083 at 8).  24 warps: the resident warps an
// SM holds at the kernels' register budgets (the fp32 forward's 32 gained
// nothing more).
static void set_lanes(VolumeArgs& a, uint64_t tiles) {
  const uint64_t resident = (uint64_t)device_sm_count_vol() * 24u;
  a.lanes = 32;
  if (a.tile_end > 1u << 29) return;  // a range's part ids stay below 2^32
  while (a.lanes > 8u && tiles * (64u / a.lanes) <= resident) a.lanes /= 2;
}

// Blocks of a launch over `tiles` tiles.
static uint32_t march_blocks(const VolumeArgs& a, uint32_t tiles) {
  constexpr uint32_t kWarps = kMarchThreads / 32;
  return (uint32_t)(((uint64_t)tiles * (32u / a.lanes) + kWarps - 1) / kWarps);
}

cudaError_t launch_volume_forward(VolumeArgs& a, cudaStream_t s) {
  const uint32_t end = a.tile_end ? a.tile_end : tile_ids(a);
  const uint32_t tiles = end > a.tile_begin ? end - a.tile_begin : 0u;
  if (tiles == 0) return cudaSuccess;
  set_lanes(a, tiles);
  const uint32_t blocks = march_blocks(a, tiles);
  const bool skip = a.v.cell_mask != nullptr;
  switch (a.v.precision) {
    case 0: launch_forward<0>(a, skip, blocks, s); break;
    case 1: launch_forward<1>(a, skip, blocks, s); break;
    case 2: launch_forward<2>(a, skip, blocks, s); break;
    case 3: launch_forward<3>(a, skip, blocks, s); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

// Edge records (GradVis) pay where the launch is bound by its atomics and the
// doubled scratch costs little.  Backward of smooth noise in trees of 128^3 and
// 512^3 voxels, ms without / with them:
//  * a scratch that leaves L2 (129 MB) turns the atomics it saves into DRAM
//    traffic.  4 M rays: 3.9 k bricks (90 MB with edges) 9.81 / 7.99; 16.8 M
//    rays: 4.9 k 8.18 / 8.09, 9.5 k (221 MB) 13.73 / 13.61, 14 k 19.4 / 19.4,
//    26 k 31.0 / 31.5, 64 k bricks 50.4 / 51.8;
//  * with few rays its zeroing and fold are not earned back.  3.9 k bricks, rays
//    per lattice point 0.04: 0.99 / 1.10, 0.09: 1.32 / 1.31, 0.19: 2.04 / 1.86.
// How many of the cells hold colour is known on the device only: where all do,
// nothing is saved (4.1 k bricks, 4 M rays 10.6 / 10.9, half of them 10.5 / 9.8).
bool backward_uses_edges(VolumeArgs& a, uint64_t rays) {
  const uint64_t points = (uint64_t)a.v.nbricks * (uint64_t)kL3;
  if (points * 32u > 128u << 20 || rays * 6u < points) return false;
  const uint32_t tiles = tile_ids(a);
  set_lanes(a, tiles);
  return !fits_small(march_blocks(a, tiles));
}

cudaError_t launch_volume_backward(VolumeArgs& a, bool edges, cudaStream_t s) {
  const uint32_t tiles = tile_ids(a);
  if (tiles == 0) return cudaSuccess;
  set_lanes(a, tiles);
  const uint32_t blocks = march_blocks(a, tiles);
  // only fp32 (learnable) volumes have an adjoint
  if (a.v.precision == 1)
    edges ? launch_backward<1, true>(a, blocks, s) : launch_backward<1, false>(a, blocks, s);
  else if (a.v.precision == 2)
    edges ? launch_backward<2, true>(a, blocks, s) : launch_backward<2, false>(a, blocks, s);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

cudaError_t launch_cell_mask(const VolumeView& v, uint32_t* mask, cudaStream_t s) {
  if (!v.nbricks) return cudaSuccess;
  const uint32_t threads = v.nbricks * 16u * 32u;
  const uint32_t blocks = (threads + 255u) / 256u;
  switch (v.precision) {
    case 0: cell_mask_kernel<0><<<blocks, 256, 0, s>>>(v, mask); break;
    case 1: cell_mask_kernel<1><<<blocks, 256, 0, s>>>(v, mask); break;
    case 2: cell_mask_kernel<2><<<blocks, 256, 0, s>>>(v, mask); break;
    default: cell_mask_kernel<3><<<blocks, 256, 0, s>>>(v, mask); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_brick_bits(const VolumeView& v, uint32_t* bits, cudaStream_t s) {
  const uint64_t n = (uint64_t)v.nb * v.nb * v.nb;
  const uint32_t nwords = (uint32_t)((n + 31) / 32);
  brick_bits_kernel<<<(uint32_t)(((uint64_t)nwords * 32 + 255) / 256), 256, 0, s>>>(v, bits,
                                                                                   nwords);
  return cudaGetLastError();
}

cudaError_t launch_apron_fold(const VolumeArgs& a, int channels, float* g, bool gather,
                              cudaStream_t s) {
  if (a.v.nbricks == 0) return cudaSuccess;
  const int blocks = 2 * device_sm_count_vol() * 8;
  if (gather) fold_gather_kernel<<<blocks, 256, 0, s>>>(a, channels, g);
  fold_scatter_kernel<<<blocks, 256, 0, s>>>(a, channels, g);
  return cudaGetLastError();
}

template <bool kEdges>
__global__ void unpack_grads_kernel(const float4* __restrict__ p, uint32_t n, float* gd,
                                    float* ga) {
  for (uint64_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const uint32_t i = (uint32_t)k;  // (k: n may be within a stride of 2^32)
    const float4 v = point_grad<kEdges>(p, i, (int)(i % (uint32_t)kL3 % (uint32_t)kL));
    gd[i] += v.w;
    ga[3 * (size_t)i] += v.x;
    ga[3 * (size_t)i + 1] += v.y;
    ga[3 * (size_t)i + 2] += v.z;
  }
}

cudaError_t launch_unpack_grads(const float4* scratch, bool edges, uint32_t n,
                                float* grad_density, float* grad_albedo, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  auto kern = edges ? unpack_grads_kernel<true> : unpack_grads_kernel<false>;
  kern<<<2 * device_sm_count_vol() * 8, 256, 0, s>>>(scratch, n, grad_density, grad_albedo);
  return cudaGetLastError();
}

__global__ void pack_f32_kernel(const float* __restrict__ d, const float* __restrict__ c,
                                uint32_t n, float4* __restrict__ out) {
  for (uint64_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = make_float4(c[3 * i], c[3 * i + 1], c[3 * i + 2], d[i]);
}

cudaError_t launch_pack_f32(const float* density, const float* albedo, uint32_t n,
                            float4* packed, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  pack_f32_kernel<<<2 * device_sm_count_vol() * 8, 256, 0, s>>>(density, albedo, n, packed);
  return cudaGetLastError();
}

// One warp per brick (blocks of 256): its 729 lattice points packed, and the
// cell occupancy mask gathered from ballots on the way.  A point whose albedo
// is not finite, or so large that interpolation could overflow, counts as set,
// so a sample the mask lets the march pass over adds exactly nothing (0 x
// albedo).
__global__ void __launch_bounds__(256) pack_train_kernel(const float* __restrict__ d,
                                                         const float* __restrict__ c,
                                                         uint32_t nbricks,
                                                         float4* __restrict__ out,
                                                         uint32_t* __restrict__ mask,
                                                         uint32_t* __restrict__ marked) {
  __shared__ uint32_t nzbits[8][24];
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t* nz = nzbits[threadIdx.x >> 5];
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < nbricks; b += nwarps) {
    const size_t base = (size_t)b * kL3;
    for (uint32_t q0 = 0; q0 < 24u; q0 += 8u) {
      float4 v[8];
#pragma unroll
      for (uint32_t u = 0; u < 8u; ++u) {
        const uint32_t k = lane + 32u * (q0 + u);
        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k < (uint32_t)kL3) {
          const float* q = c + 3 * (base + k);
          v[u] = make_float4(__ldg(q), __ldg(q + 1), __ldg(q + 2), __ldg(d + base + k));
        }
      }
#pragma unroll
      for (uint32_t u = 0; u < 8u; ++u) {
        const uint32_t k = lane + 32u * (q0 + u);
        if (k < (uint32_t)kL3) out[base + k] = v[u];
        const bool set = v[u].w != 0.f || !(fabsf(v[u].x) <= 1e38f) ||
                         !(fabsf(v[u].y) <= 1e38f) || !(fabsf(v[u].z) <= 1e38f);
        const uint32_t bits = __ballot_sync(0xFFFFFFFFu, set);
        if (lane == 0) nz[q0 + u] = bits;
      }
    }
    __syncwarp();
    const uint32_t word = lane < 16u ? cell_mask_word(nz, lane) : 0u;
    if (lane < 16u) mask[(size_t)b * 16u + lane] = word;
    const uint32_t n = __reduce_add_sync(0xFFFFFFFFu, __popc(word));
    if (lane == 0) marked[b] = n;
    __syncwarp();
  }
}

cudaError_t launch_pack_train(const float* density, const float* albedo, uint32_t nbricks,
                              float4* packed, uint32_t* mask, uint32_t* marked, cudaStream_t s) {
  if (nbricks == 0) return cudaSuccess;
  const uint32_t blocks = (nbricks + 7u) / 8u, cap = (uint32_t)device_sm_count_vol() * 16u;
  pack_train_kernel<<<blocks < cap ? blocks : cap, 256, 0, s>>>(density, albedo, nbricks, packed,
                                                               mask, marked);
  return cudaGetLastError();
}

// Unpack and apron fold in one pass over the lattice points: a point's owner
// (its own brick, or the upper neighbour for an apron point) sums its copies in
// the order of fold_gather_kernel.  Interior points have one copy and need no
// neighbour.  3072 bricks: 14 us, 27 from edge records, where an unpack, two
// gathers, two scatters and the zeroing of two tensors took 105.
template <bool kEdges>
__global__ void __launch_bounds__(256) fold_grads_kernel(const float4* __restrict__ p,
                                                         const int32_t* __restrict__ up,
                                                         const int32_t* __restrict__ dn,
                                                         uint32_t npoints,
                                                         float* __restrict__ gd,
                                                         float* __restrict__ ga) {
  for (uint64_t k = blockIdx.x * blockDim.x + threadIdx.x; k < npoints;
       k += gridDim.x * blockDim.x) {
    const uint32_t i = (uint32_t)k;  // (k: npoints may be within a stride of 2^32)
    const uint32_t b = i / (uint32_t)kL3, q = i % (uint32_t)kL3;
    int x = (int)(q % kL), y = (int)((q / kL) % kL), z = (int)(q / (kL * kL));
    const int m0 = (x == 8) | ((y == 8) << 1) | ((z == 8) << 2);
    int own = (int)b;
    if (m0) {
      own = __ldg(up + (size_t)b * 7 + (m0 - 1));
      x &= 7;
      y &= 7;
      z &= 7;
    }
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (own >= 0) {
      v = point_grad<kEdges>(p, (size_t)own * kL3 + (size_t)((z * kL + y) * kL + x), x);
      if (x == 0 || y == 0 || z == 0) {
        for (int m = 1; m < 8; ++m) {
          const int dx = m & 1, dy = (m >> 1) & 1, dz = m >> 2;
          if ((dx && x) || (dy && y) || (dz && z)) continue;
          const int nb = __ldg(dn + (size_t)own * 7 + (m - 1));
          if (nb < 0) continue;
          const float4 c = point_grad<kEdges>(
              p,
              (size_t)nb * kL3 +
                  (size_t)(((z + 8 * dz) * kL + (y + 8 * dy)) * kL + (x + 8 * dx)),
              x + 8 * dx);
          v.x += c.x;
          v.y += c.y;
          v.z += c.z;
          v.w += c.w;
        }
      }
    }
    gd[i] = v.w;
    ga[3 * (size_t)i] = v.x;
    ga[3 * (size_t)i + 1] = v.y;
    ga[3 * (size_t)i + 2] = v.z;
  }
}

cudaError_t launch_fold_grads(const VolumeArgs& a, const float4* scratch, bool edges,
                              float* grad_density, float* grad_albedo, cudaStream_t s) {
  const uint32_t n = a.v.nbricks * (uint32_t)kL3;
  if (n == 0) return cudaSuccess;
  const uint32_t blocks = (n + 255u) / 256u, cap = (uint32_t)device_sm_count_vol() * 32u;
  auto kern = edges ? fold_grads_kernel<true> : fold_grads_kernel<false>;
  kern<<<blocks < cap ? blocks : cap, 256, 0, s>>>(scratch, a.nbr_up, a.nbr_dn, n, grad_density,
                                                  grad_albedo);
  return cudaGetLastError();
}

int device_sm_count_vol() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
    n = 1;
  return n;
}

}  // namespace yv
