// svo_build.cu - GPU build of the canonical sparse voxel octree from a
// dense density grid: the iso/raw-source form of DynamicSVO::BuildRange
// (the GROW pass driven by a voxel source, ore/src/main.cpp:37-129,
// demo/Demo.cpp:82-114; the DynamicSVO source is not in the reference
// snapshot), with the surface-voxel rule of scene_gen.py:32-66 and the
// VoxNode layout of reaction/report/main.tex:36-56.
//
// Rules (identical to the host generators' canonical form):
//   voxel v of the 2^depth grid is solid iff density[v] > iso; a solid voxel
//   with a 6-neighbour outside the grid or not solid is a surface voxel (a
//   leaf); a cube region without surface voxels is EmptyNode (no solid
//   voxel) or FullNode; nodes are numbered breadth-first from the root
//   (id 0), children in child order c = x | y<<1 | z<<2, leaves in the same
//   order.  Leaf: RGB of the voxel (white without an rgb grid), A = 255,
//   normal = quantised normalize of the central difference (d(x-1) -
//   d(x+1), ...) with coordinates clamped to the grid, every step an FP32
//   round-to-nearest operation (zero for a zero or non-finite length).
//
// GB300 design, bit-parallel with no list of regions: breadth-first order with
// children in x | y<<1 | z<<2 order is the Morton order of a level's regions,
// so every level is two bit arrays in Morton order, `node` and `full`, and
//   - byte r of level k+1's arrays holds the 8 children of region r of level k;
//   - a node's number is the count of node bits before its own, over the
//     levels from the root down; its first node child is the count at its
//     child byte.
//   1. one pass packs the solid bits of the grid (row words);
//   2. a warp per 128 x 8 x 8 voxels finds the surface voxels by bit shifts and
//      writes the node and full words (64 regions of 2^3 voxels = 8^3 voxels
//      each) and their leaf counts;
//   3. byte-wise folds give the levels above, prefix sums over the words of all
//      levels number the nodes, another the leaves; the host reads two totals;
//   4. a warp per word writes its nodes; at the bottom one finds the surface
//      voxels again and writes their leaves.  The outputs are the VoxNodes and
//      attributes of the host container or the renderer's own records.
// Depth <= 11 (a 2048^3 grid: 8.6 G voxels, 34 GB of float density).
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "dev_scan.cuh"
#include "yv_internal.h"
#include "yv_kernels.h"

namespace yv {
namespace {

struct Grid {
  const float* d;
  const uint8_t* rgb;
  int G;
  float iso;
};

__device__ __forceinline__ size_t vidx(int G, int x, int y, int z) {
  return (size_t)x + (size_t)G * ((size_t)y + (size_t)G * (size_t)z);
}

__device__ __forceinline__ float dens_clamped(const Grid& g, int x, int y, int z) {
  x = x < 0 ? 0 : (x >= g.G ? g.G - 1 : x);
  y = y < 0 ? 0 : (y >= g.G ? g.G - 1 : y);
  z = z < 0 ? 0 : (z >= g.G ? g.G - 1 : z);
  return __ldg(g.d + vidx(g.G, x, y, z));
}

// Pass 1a: solid bits, one 32-voxel run of a row per warp and word (lane i
// tests x = 32 w + i, a ballot packs the run): S[(z G + y) WR + w],
// WR = max(1, G / 32) words per row (a power of two, as is G); bits beyond
// the grid are 0.  Eight words per iteration keep eight coalesced 128-byte
// loads in flight; word indices fit 32 bits (G^2 WR <= 2^28) and are split
// with shifts.
__global__ void solid_bits_kernel(Grid g, uint32_t WR, uint32_t* S) {
  constexpr int kU = 8;
  const uint32_t lane = threadIdx.x & 31u;
  const int wsh = __ffs(WR) - 1;
  const uint32_t total = (uint32_t)g.G * (uint32_t)g.G * WR;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w0 < total;
       w0 += kU * nwarps) {
    bool sol[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint32_t wi = w0 + (uint32_t)u * nwarps;
      const uint32_t x = ((wi & (WR - 1u)) << 5) + lane;
      sol[u] = wi < total && x < (uint32_t)g.G &&
               __ldg(g.d + (uint64_t)(wi >> wsh) * (uint64_t)g.G + x) > g.iso;
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint32_t wi = w0 + (uint32_t)u * nwarps;
      const uint32_t m = __ballot_sync(0xFFFFFFFFu, sol[u]);
      if (lane == 0 && wi < total) S[wi] = m;
    }
  }
}

// Pass 1a for rows of 128 voxels or more (G >= 128) of a grid that starts on
// a 16-byte boundary: one 128-voxel chunk per warp and iteration, each lane a
// 16-byte load of 4 voxels; the lanes' 4-bit groups are ORed into 32-bit words
// within groups of 8 lanes (3 shuffles), lane 8j writing word j of the chunk.
// Same bits as above.
__global__ void solid_bits_v4_kernel(Grid g, uint32_t WR, uint32_t* S) {
  constexpr int kU = 4;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t CR = WR >> 2;  // chunks per row
  const int csh = __ffs(CR) - 1;
  const uint32_t total = (uint32_t)g.G * CR * (uint32_t)g.G;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const float4* d4 = reinterpret_cast<const float4*>(g.d);
  for (uint32_t c0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c0 < total;
       c0 += kU * nwarps) {
    float4 v[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint32_t c = c0 + (uint32_t)u * nwarps;
      v[u] = c < total ? __ldg(d4 + (((uint64_t)(c >> csh) * g.G + ((c & (CR - 1u)) << 7)) >> 2) +
                               lane)
                       : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint32_t c = c0 + (uint32_t)u * nwarps;
      const uint32_t nib = (uint32_t)(v[u].x > g.iso) | ((uint32_t)(v[u].y > g.iso) << 1) |
                           ((uint32_t)(v[u].z > g.iso) << 2) | ((uint32_t)(v[u].w > g.iso) << 3);
      uint32_t word = nib << (4 * (lane & 7u));
      word |= __shfl_xor_sync(0xFFFFFFFFu, word, 1);
      word |= __shfl_xor_sync(0xFFFFFFFFu, word, 2);
      word |= __shfl_xor_sync(0xFFFFFFFFu, word, 4);
      if ((lane & 7u) == 0u && c < total)
        S[((uint64_t)(c >> csh) * WR) + ((c & (CR - 1u)) << 2) + (lane >> 3)] = word;
    }
  }
}

// 10-bit spread of a block coordinate: bit i to bit 3 i.
__device__ __forceinline__ uint32_t spread3(uint32_t v) {
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  return (v | (v << 2)) & 0x09249249u;
}
// Word w of row (y, z) of the solid bits, 0 outside the grid.
__device__ __forceinline__ uint32_t solid_word(const uint32_t* S, int G, int WR, int w, int y,
                                               int z) {
  if (w < 0 || w >= WR || y < 0 || y >= G || z < 0 || z >= G) return 0u;
  return __ldg(S + ((uint64_t)z * (uint64_t)G + (uint64_t)y) * (uint64_t)WR + (uint64_t)w);
}

// A warp's share of the two passes over the solid bits: 4 words x 8 x 8 rows
// (16 blocks of 8^3 voxels), lane = word | y << 2, the 8 rows of a lane's word
// along z in registers.  Its loads are 16 bytes of a row for 4 lanes; a layout
// of one word x 64 rows a warp reads a line per lane (1024^3: 198 and 246 us
// for the two passes), a tile in shared memory took 249 and 437 us.
struct BitRows {
  uint32_t W[10];    // solid bits of rows z0 - 1 .. z0 + 8
  uint32_t surf[8];  // surface bits of rows z0 .. z0 + 7
};

// The warp's place: word of the lane, block row and column.
__device__ __forceinline__ bool rows_place(int WR, uint32_t nbl, int& w, uint32_t& BY,
                                           uint32_t& BZ) {
  const uint32_t groups = ((uint32_t)WR + 3u) / 4u;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  w = (int)(4u * (warp % groups) + (threadIdx.x & 3u));
  BY = (warp / groups) % nbl;
  BZ = warp / (groups * nbl);
  return BZ < nbl;
}

// The solid bits; false (for the whole warp): none of the 8 rows has any.
__device__ __forceinline__ bool load_rows(BitRows& t, const uint32_t* S, int G, int WR, int w,
                                          int y, int z0) {
#pragma unroll
  for (int k = 0; k < 10; ++k) t.W[k] = solid_word(S, G, WR, w, y, z0 + k - 1);
  uint32_t any = 0;
#pragma unroll
  for (int k = 1; k < 9; ++k) any |= t.W[k];
  return __any_sync(0xFFFFFFFFu, any != 0u) != 0;
}

// Surface bits: solid with a 6-neighbour that is not (outside the grid nothing
// is solid).
__device__ __forceinline__ void surface_rows(BitRows& t, const uint32_t* S, int G, int WR, int w,
                                             int y, int z0, uint32_t lane) {
  const uint32_t wl = lane & 3u, yl = lane >> 2;
  uint32_t hx[8], hy[8];  // rows beyond the warp's words and rows
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    hx[k] = (wl == 0u || wl == 3u) ? solid_word(S, G, WR, wl ? w + 1 : w - 1, y, z0 + k) : 0u;
    hy[k] = (yl == 0u || yl == 7u) ? solid_word(S, G, WR, w, yl ? y + 1 : y - 1, z0 + k) : 0u;
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t c = t.W[k + 1];
    const uint32_t l = __shfl_up_sync(0xFFFFFFFFu, c, 1), r = __shfl_down_sync(0xFFFFFFFFu, c, 1);
    const uint32_t d = __shfl_up_sync(0xFFFFFFFFu, c, 4), u = __shfl_down_sync(0xFFFFFFFFu, c, 4);
    const uint32_t lx = __funnelshift_l(wl == 0u ? hx[k] : l, c, 1),
                   rx = __funnelshift_r(c, wl == 3u ? hx[k] : r, 1);
    t.surf[k] = c & ~(lx & rx & (yl == 0u ? hy[k] : d) & (yl == 7u ? hy[k] : u) & t.W[k] &
                      t.W[k + 2]);
  }
}

// Pass 2: node and full words of the bottom regions, in Morton order, and the
// leaves (surface voxels) of each word.  1024^3: per-region classes and codes
// took 187 us and 400 MB, the node and full bits are 17 MB each.
__global__ void __launch_bounds__(256) classify_kernel(const uint32_t* S, int G, int WR,
                                                       uint64_t* node, uint64_t* full,
                                                       uint16_t* leaves) {
  const uint32_t lane = threadIdx.x & 31u, yl = lane >> 2;
  const uint32_t nbl = (uint32_t)(G + 7) / 8u;  // 8^3 blocks per axis
  int w;
  uint32_t BY, BZ;
  if (!rows_place(WR, nbl, w, BY, BZ)) return;
  const int y = (int)(8u * BY + yl), z0 = (int)(8u * BZ);
  BitRows t;
  // words of the lane's 4 blocks, lower and upper half, and leaf counts (two
  // blocks to a register)
  uint32_t n[4][2] = {}, f[4][2] = {}, lf[2] = {};
  if (load_rows(t, S, G, WR, w, y, z0)) {
    surface_rows(t, S, G, WR, w, y, z0, lane);
    // a region's bit in the Morton order of its block: x bits 0 and 3, y 1
    // and 4, z 2 and 5 (the upper half)
    const uint32_t shy = 2u * ((yl >> 1) & 1u) + 16u * (yl >> 2);
#pragma unroll
    for (int rz = 0; rz < 4; ++rz) {
      const uint32_t s0 = t.surf[2 * rz], s1 = t.surf[2 * rz + 1];
      uint32_t any = t.W[2 * rz + 1] | t.W[2 * rz + 2];
      uint32_t fu = (t.W[2 * rz + 1] & ~s0) & (t.W[2 * rz + 2] & ~s1);
      any |= __shfl_xor_sync(0xFFFFFFFFu, any, 4);
      fu &= __shfl_xor_sync(0xFFFFFFFFu, fu, 4);
      any = (any | (any >> 1)) & 0x55555555u;  // bit 2 rx: region (rx, y / 2, rz)
      fu = fu & (fu >> 1) & 0x55555555u;
      // bits 0, 2, 4, 6 of each byte to its bits 0, 1 and 8, 9 of a half word:
      // first to 0, 1, 4, 5
      uint32_t a = any & ~fu, b = fu;
      a = (a & 0x11111111u) | ((a >> 1) & 0x22222222u);
      b = (b & 0x11111111u) | ((b >> 1) & 0x22222222u);
      const uint32_t sh = shy + 4u * (uint32_t)(rz & 1);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t va = (a >> (8 * j)) & 0xFFu, vb = (b >> (8 * j)) & 0xFFu;
        n[j][rz >> 1] |= ((va | (va << 4)) & 0x303u) << sh;
        f[j][rz >> 1] |= ((vb | (vb << 4)) & 0x303u) << sh;
        lf[j >> 1] += (uint32_t)(__popc(s0 & (0xFFu << (8 * j))) +
                                 __popc(s1 & (0xFFu << (8 * j))))
                      << (16 * (j & 1));
      }
    }
    // over the rows y (a pair of rows holds the same regions)
#pragma unroll
    for (int o = 8; o <= 16; o <<= 1)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          n[j][h] |= __shfl_xor_sync(0xFFFFFFFFu, n[j][h], o);
          f[j][h] |= __shfl_xor_sync(0xFFFFFFFFu, f[j][h], o);
        }
#pragma unroll
    for (int o = 4; o <= 16; o <<= 1)
#pragma unroll
      for (int h = 0; h < 2; ++h) lf[h] += __shfl_xor_sync(0xFFFFFFFFu, lf[h], o);
  }
  // lane (word, yl): block yl of the word, for yl < 4
  const uint32_t BX = 4u * (uint32_t)w + yl;
  if (yl < 4u && BX < nbl) {
    const uint32_t m = spread3(BX) | (spread3(BY) << 1) | (spread3(BZ) << 2);
    uint32_t nl = n[0][0], nh = n[0][1], fl = f[0][0], fh = f[0][1];
#pragma unroll
    for (uint32_t j = 1; j < 4u; ++j)
      if (yl == j) {
        nl = n[j][0];
        nh = n[j][1];
        fl = f[j][0];
        fh = f[j][1];
      }
    node[m] = (uint64_t)nl | ((uint64_t)nh << 32);
    full[m] = (uint64_t)fl | ((uint64_t)fh << 32);
    leaves[m] = (uint16_t)((yl < 2u ? lf[0] : lf[1]) >> (16u * (yl & 1u)));
  }
}

// Level k's node and full bits of the 8 regions whose children are the bytes
// of words nw, fw of level k+1: EMPTY if all 8 children are, FULL if all 8
// are, else a node.
__device__ __forceinline__ void fold_word(uint64_t nw, uint64_t fw, uint8_t& node, uint8_t& full) {
  constexpr uint64_t k7F = 0x7F7F7F7F7F7F7F7Full, k80 = ~k7F;
  const uint64_t t = nw | fw, u = ~fw;
  const uint64_t some = (((t & k7F) + k7F) | t) & k80;       // bytes that are not 0
  const uint64_t part = (((u & k7F) + k7F) | u) & k80;       // bytes of fw that are not 0xFF
  // bits 7, 15, ... of a word gathered into a byte
  constexpr uint64_t kGather = 0x0002040810204081ull;
  node = (uint8_t)(((some & part) >> 7) * (kGather << 7) >> 56);
  full = (uint8_t)(((~part & k80) >> 7) * (kGather << 7) >> 56);
}

// Words of level k (64 regions each, at least one).
__host__ __device__ __forceinline__ uint32_t level_words(int k) {
  return k < 2 ? 1u : 1u << (3 * k - 6);
}

// Pass 3a: the bytes `node` and `full` of level k from the words cn, cf of level
// k+1 (a word holds the children of 8 regions).
__global__ void fold_kernel(const uint64_t* cn, const uint64_t* cf, uint32_t words, uint8_t* node,
                            uint8_t* full) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < words) fold_word(cn[i], cf[i], node[i], full[i]);
}

// Levels k_top..0 in one block.
__global__ void __launch_bounds__(1024) fold_top_kernel(uint64_t* node, uint64_t* full,
                                                        int k_top) {
  uint32_t at = 0;  // first word of level k + 1
  for (int k = 0; k <= k_top; ++k) at += level_words(k);
  for (int k = k_top; k >= 0; --k) {
    const uint32_t words = level_words(k + 1), to = at - level_words(k);
    for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) {
      uint8_t n, f;
      fold_word(node[at + i], full[at + i], n, f);
      reinterpret_cast<uint8_t*>(node + to)[i] = n;
      reinterpret_cast<uint8_t*>(full + to)[i] = f;
    }
    __syncthreads();
    at = to;
  }
}

// Pass 3b: prefix sums of the node bits over the words of all levels and of
// the leaf counts over the bottom words, in chunks: sums per chunk (first the
// node chunks, then the leaf chunks), their scan in one block each, the words.
constexpr uint32_t kChunk = 2048;  // words: 256 threads x 8

__device__ __forceinline__ uint32_t word_count(const uint64_t* node, const uint16_t* leaves,
                                               bool is_leaf, uint32_t i) {
  return is_leaf ? (uint32_t)leaves[i] : (uint32_t)__popcll(node[i]);
}

__global__ void __launch_bounds__(256) chunk_sums_kernel(const uint64_t* node, uint32_t nwords,
                                                         uint32_t nchunks, const uint16_t* leaves,
                                                         uint32_t lwords, uint32_t* sums) {
  __shared__ uint32_t tot;
  const bool lf = blockIdx.x >= nchunks;
  const uint32_t c = lf ? blockIdx.x - nchunks : blockIdx.x, n = lf ? lwords : nwords;
  if (threadIdx.x == 0) tot = 0;
  __syncthreads();
  uint32_t t = 0;
#pragma unroll
  for (uint32_t k = 0; k < 8u; ++k) {
    const uint32_t i = c * kChunk + k * 256u + threadIdx.x;
    if (i < n) t += word_count(node, leaves, lf, i);
  }
  t = __reduce_add_sync(0xFFFFFFFFu, t);
  if ((threadIdx.x & 31u) == 0 && t) atomicAdd(&tot, t);
  __syncthreads();
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// Inclusive scan of v over a block of n warps; warp_tot: n words of shared
// memory.  Returns the inclusive sum, *total the block's.
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* warp_tot, uint32_t nwarps,
                                               uint32_t* total) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, v, o);
    if (lane >= (uint32_t)o) v += u;
  }
  if (lane == 31) warp_tot[warp] = v;
  __syncthreads();
  uint32_t before = 0, all = 0;
  for (uint32_t w = 0; w < nwarps; ++w) {
    if (w < warp) before += warp_tot[w];
    all += warp_tot[w];
  }
  __syncthreads();
  *total = all;
  return v + before;
}

// sums -> exclusive prefix, in place; totals[block] = all.  Block 0: the
// nodes, block 1: the leaves.
__global__ void __launch_bounds__(1024) chunk_scan_kernel(uint32_t* sums, uint32_t nchunks,
                                                          uint32_t lchunks, uint32_t* totals) {
  __shared__ uint32_t warp_tot[32];
  uint32_t* p = blockIdx.x ? sums + nchunks : sums;
  const uint32_t n = blockIdx.x ? lchunks : nchunks;
  uint32_t run = 0;
  for (uint32_t i0 = 0; i0 < n; i0 += 1024u) {
    const uint32_t i = i0 + threadIdx.x, v = i < n ? p[i] : 0u;
    uint32_t all;
    const uint32_t inc = block_scan(v, warp_tot, 32u, &all);
    if (i < n) p[i] = run + inc - v;
    run += all;
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = run;
}

__global__ void __launch_bounds__(256) prefix_kernel(const uint64_t* node, uint32_t nwords,
                                                     uint32_t nchunks, const uint16_t* leaves,
                                                     uint32_t lwords, const uint32_t* sums,
                                                     uint32_t* node_pre, uint32_t* leaf_pre) {
  __shared__ uint32_t warp_tot[8];
  const bool lf = blockIdx.x >= nchunks;
  const uint32_t c = lf ? blockIdx.x - nchunks : blockIdx.x, n = lf ? lwords : nwords;
  uint32_t* out = lf ? leaf_pre : node_pre;
  const uint32_t i0 = c * kChunk + 8u * threadIdx.x;
  uint32_t v[8], t = 0, all;
#pragma unroll
  for (uint32_t k = 0; k < 8u; ++k) {
    v[k] = i0 + k < n ? word_count(node, leaves, lf, i0 + k) : 0u;
    t += v[k];
  }
  uint32_t run = sums[blockIdx.x] + block_scan(t, warp_tot, 8u, &all) - t;
#pragma unroll
  for (uint32_t k = 0; k < 8u; ++k) {
    if (i0 + k < n) out[i0 + k] = run;
    run += v[k];
  }
}

// Where the nodes and leaves go: the host container's pool (nodes, attrs) or
// the renderer's records (rec, cold, shade).
struct BuildOut {
  yv_vox_node* nodes;
  yv_leaf_attr* attrs;
  uint2* rec;
  uint2* cold;
  uint4* shade;
};

// Node `id`: children of mask `nm` are nodes from `first` on or (leaf) leaves
// from `first` on; of the others those of `fm` are full.
template <bool kHost, bool kLeaf>
__device__ __forceinline__ void write_node(const BuildOut& o, uint32_t id, uint32_t nm,
                                           uint32_t fm, uint32_t first) {
  if (kHost) {
    yv_vox_node v;
    v.flags = kLeaf ? nm | ((~nm & 0xFFu) << 8) : (~nm & 0xFFu) << 8;
    v.data = 0;
    uint32_t next = first;
#pragma unroll
    for (int c = 0; c < 8; ++c)
      v.child[c] = ((nm >> c) & 1u) ? next++
                                    : (((fm >> c) & 1u) ? YV_FULL_NODE : YV_EMPTY_NODE);
    o.nodes[id] = v;
  } else {
    uint32_t codes = 0, rank = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      uint32_t k = YV_CODE_NULL;
      if ((nm >> c) & 1u) k = kLeaf ? YV_CODE_LEAF : rank++;
      codes |= k << (28 - 4 * c);
    }
    o.rec[id] = make_uint2(kLeaf ? 0u : first, codes);
    o.cold[id] = make_uint2(id, kLeaf ? first : 0u);
  }
}

// Pass 4a: the nodes above the bottom (words [0, nwords) of all levels but the
// last), a thread per byte: 8 regions, whose children are one word of the next
// level (the 8 words of a word's children start at 8 x its place there).
template <bool kHost>
__global__ void __launch_bounds__(256) emit_nodes_kernel(const uint64_t* node,
                                                         const uint64_t* full,
                                                         const uint32_t* pre, uint32_t nwords,
                                                         BuildOut out) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, i = t >> 3, h = t & 7u;
  if (i >= nwords) return;
  const uint64_t nw = node[i];
  uint32_t todo = (uint32_t)(nw >> (8u * h)) & 0xFFu;
  if (!todo) return;
  uint32_t at = 0;  // the word's level and its first word
  int k = 0;
  while (i >= at + level_words(k)) at += level_words(k++);
  // (levels 0 and 1 hold fewer than 64 regions: only their first byte is set)
  const uint32_t cw = at + level_words(k) + 8u * (i - at) + h;
  const uint64_t cn = node[cw], cf = full[cw];
  uint32_t id = pre[i] + (uint32_t)__popcll(nw & ((1ull << (8u * h)) - 1ull));
  uint32_t first = pre[cw];
  for (uint32_t c = 0; c < 8u; ++c) {
    const uint32_t nm = (uint32_t)(cn >> (8u * c)) & 0xFFu;
    if ((todo >> c) & 1u)
      write_node<kHost, false>(out, id++, nm, (uint32_t)(cf >> (8u * c)) & 0xFFu, first);
    first += (uint32_t)__popc(nm);
  }
}

__device__ __forceinline__ int8_t quant_n(float v) {
  float q = floorf(__fadd_rn(__fmul_rn(127.f, v), 0.5f));
  if (q > 127.f) q = 127.f;
  if (q < -127.f) q = -127.f;
  return (int8_t)(int)q;
}

// Attribute of leaf voxel (x, y, z).
__device__ __forceinline__ yv_leaf_attr leaf_attr(const Grid& g, int x, int y, int z) {
  yv_leaf_attr a;
  if (g.rgb) {
    const size_t o = 3 * vidx(g.G, x, y, z);
    a.r = g.rgb[o];
    a.g = g.rgb[o + 1];
    a.b = g.rgb[o + 2];
  } else {
    a.r = a.g = a.b = 255;
  }
  a.a = 255;
  const float fx = __fsub_rn(dens_clamped(g, x - 1, y, z), dens_clamped(g, x + 1, y, z));
  const float fy = __fsub_rn(dens_clamped(g, x, y - 1, z), dens_clamped(g, x, y + 1, z));
  const float fz = __fsub_rn(dens_clamped(g, x, y, z - 1), dens_clamped(g, x, y, z + 1));
  const float len2 =
      __fadd_rn(__fadd_rn(__fmul_rn(fx, fx), __fmul_rn(fy, fy)), __fmul_rn(fz, fz));
  float nx = 0.f, ny = 0.f, nz = 0.f;
  if (len2 > 0.f && len2 <= 3.402823466e38f) {
    const float len = __fsqrt_rn(len2);
    nx = __fdiv_rn(fx, len);
    ny = __fdiv_rn(fy, len);
    nz = __fdiv_rn(fz, len);
  }
  a.nx = quant_n(nx);
  a.ny = quant_n(ny);
  a.nz = quant_n(nz);
  a.nw = 0;
  return a;
}

// The renderer's 16-byte shading record of an attribute (RGBA8 + unit normal,
// the FP32 normalisation of the upload path).
__device__ __forceinline__ uint4 shade_record(const yv_leaf_attr& a) {
  const float nx = (float)a.nx, ny = (float)a.ny, nz = (float)a.nz;
  const float len2 =
      __fadd_rn(__fadd_rn(__fmul_rn(nx, nx), __fmul_rn(ny, ny)), __fmul_rn(nz, nz));
  float u[3] = {0.f, 0.f, 0.f};
  if (len2 > 0.f) {
    const float len = __fsqrt_rn(len2);
    u[0] = __fdiv_rn(nx, len);
    u[1] = __fdiv_rn(ny, len);
    u[2] = __fdiv_rn(nz, len);
  }
  return make_uint4((uint32_t)a.r | ((uint32_t)a.g << 8) | ((uint32_t)a.b << 16) |
                        ((uint32_t)a.a << 24),
                    __float_as_uint(u[0]), __float_as_uint(u[1]), __float_as_uint(u[2]));
}

// Pass 4b: bottom nodes and leaves.  A warp takes those of its 16 blocks that
// have a node one after the other: the surface bits of their 64 rows again, a
// lane per region writes its node and lists its leaf voxels in order, then the
// lanes take the leaves 32 at a time (the density loads of neighbouring leaves
// share sectors).  Blocks of one warp: what warps find differs (build and
// frame of 1024^3 spheres 1253 us, 1320 with 8 warps a block).
template <bool kHost>
__global__ void __launch_bounds__(32) emit_bottom_kernel(Grid g, const uint32_t* S, int WR,
                                                          const uint64_t* node,
                                                          const uint32_t* node_pre,
                                                          const uint32_t* leaf_pre,
                                                          BuildOut out) {
  // rows z * 8 + y of the warp's 4 words
  __shared__ uint32_t s_surf[4][65], s_sol[4][65];
  __shared__ uint16_t s_leaf[512];  // x | y << 3 | z << 6 in the block
  const uint32_t lane = threadIdx.x & 31u, yl = lane >> 2;
  const uint32_t nbl = (uint32_t)(g.G + 7) / 8u;
  int w;
  uint32_t BY, BZ;
  if (!rows_place(WR, nbl, w, BY, BZ)) return;
  const uint32_t m0 = (spread3(BY) << 1) | (spread3(BZ) << 2);
  // lane (word, yl < 4): block yl of the word
  const uint32_t myBX = 4u * (uint32_t)w + yl;
  uint32_t todo = __ballot_sync(0xFFFFFFFFu, yl < 4u && myBX < nbl &&
                                                 node[m0 | spread3(myBX)] != 0ull);
  if (!todo) return;
  {
    BitRows t;
    const int y = (int)(8u * BY + yl), z0 = (int)(8u * BZ);
    load_rows(t, S, g.G, WR, w, y, z0);
    surface_rows(t, S, g.G, WR, w, y, z0, lane);
#pragma unroll
    for (uint32_t k = 0; k < 8u; ++k) {
      s_surf[lane & 3u][8u * k + yl] = t.surf[k];
      s_sol[lane & 3u][8u * k + yl] = t.W[k + 1];
    }
  }
  __syncwarp();
  const uint32_t w0 = (uint32_t)w & ~3u;
  while (todo) {
    const uint32_t l = (uint32_t)__ffs(todo) - 1u, wl = l & 3u, sh = 8u * (l >> 2);
    todo &= todo - 1u;
    const uint32_t BX = 4u * (w0 + wl) + (l >> 2), i = m0 | spread3(BX);
    const uint64_t nw = node[i];
    uint32_t nleaf = 0;  // leaves of the regions before this half
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
      const uint32_t r = lane + 32u * h;
      const uint32_t rx = (r & 1u) | ((r >> 2) & 2u), ry = ((r >> 1) & 1u) | ((r >> 3) & 2u),
                     rz = ((r >> 2) & 1u) | ((r >> 4) & 2u);
      uint32_t lm = 0, sm = 0;
#pragma unroll
      for (uint32_t q = 0; q < 4u; ++q) {
        const uint32_t row = (2u * rz + (q >> 1)) * 8u + 2u * ry + (q & 1u);
        lm |= ((s_surf[wl][row] >> (sh + 2u * rx)) & 3u) << (2u * q);
        sm |= ((s_sol[wl][row] >> (sh + 2u * rx)) & 3u) << (2u * q);
      }
      const bool in = (nw >> r) & 1ull;
      uint32_t inc = in ? (uint32_t)__popc(lm) : 0u;
      const uint32_t own = inc;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= (uint32_t)o) inc += u;
      }
      uint32_t at = nleaf + inc - own;
      nleaf += __shfl_sync(0xFFFFFFFFu, inc, 31);
      if (in) {
        write_node<kHost, true>(out, node_pre[i] + (uint32_t)__popcll(nw & ((1ull << r) - 1ull)),
                                lm, sm & ~lm, leaf_pre[i] + at);
        for (uint32_t m = lm; m; m &= m - 1u) {
          const uint32_t c = (uint32_t)__ffs(m) - 1u;
          s_leaf[at++] = (uint16_t)((2u * rx + (c & 1u)) | ((2u * ry + ((c >> 1) & 1u)) << 3) |
                                        ((2u * rz + (c >> 2)) << 6));
        }
      }
    }
    __syncwarp();
    const size_t leaf0 = leaf_pre[i];
    for (uint32_t t = lane; t < nleaf; t += 32u) {
      const uint32_t v = s_leaf[t];
      const yv_leaf_attr a = leaf_attr(g, (int)(8u * BX + (v & 7u)),
                                       (int)(8u * BY + ((v >> 3) & 7u)), (int)(8u * BZ + (v >> 6)));
      if (kHost)
        out.attrs[leaf0 + t] = a;
      else
        out.shade[leaf0 + t] = shade_record(a);
    }
    __syncwarp();
  }
}

yv_status build_fail(cudaError_t e, const char* what) {
  set_last_error(std::string("dense SVO build: ") + what + ": " + cudaGetErrorString(e));
  cudaGetLastError();
  return e == cudaErrorMemoryAllocation ? YV_ERR_OUT_OF_MEMORY : YV_ERR_CUDA;
}

// A counted tree: everything the emit passes read, in one scratch allocation.
struct SvoBuild {
  DevBuf mem;
  Grid g{};
  int depth = 0;
  uint32_t WR = 1, nwords = 0, bottom = 0;  // words of all levels; first bottom word
  uint32_t* S = nullptr;
  uint64_t *node = nullptr, *full = nullptr;
  uint32_t *node_pre = nullptr, *leaf_pre = nullptr;
  uint32_t nn = 0, na = 0, root = YV_EMPTY_NODE;
};

// Blocks of the passes over the solid bits (rows_place).
unsigned rows_blocks(const SvoBuild& b) {
  const uint64_t nbl = (uint64_t)(b.g.G + 7) / 8u;
  return (unsigned)(((b.WR + 3u) / 4u * nbl * nbl + 7u) / 8u);
}

yv_status count_dense(const float* density, const uint8_t* rgb, int depth, float iso,
                      cudaStream_t s, SvoBuild& b) {
  if (!density || depth < 1 || depth > 11 || std::isnan(iso)) return YV_ERR_INVALID_ARG;
  const int G = 1 << depth;
  b.g = Grid{density, rgb, G, iso};
  b.depth = depth;
  b.WR = G >= 32 ? (uint32_t)(G / 32) : 1u;
  const uint32_t lwords = level_words(depth - 1);
  for (int k = 0; k < depth - 1; ++k) b.bottom += level_words(k);
  b.nwords = b.bottom + lwords;
  const uint32_t nchunks = (b.nwords + kChunk - 1) / kChunk,
                 lchunks = (lwords + kChunk - 1) / kChunk;
  uint64_t total = 0;
  auto part = [&](uint64_t bytes) {
    const uint64_t at = total;
    total += (bytes + 255u) & ~255ull;
    return at;
  };
  // (the word arrays run 8 words on: levels 0 and 1 have fewer than 8 child
  // words)
  const uint64_t node_at = part((b.nwords + 8ull) * 8), full_at = part((b.nwords + 8ull) * 8),
                 np_at = part((b.nwords + 8ull) * 4), lp_at = part(lwords * 4ull),
                 lc_at = part(lwords * 2ull), sums_at = part((nchunks + (uint64_t)lchunks) * 4),
                 tot_at = part(16), S_at = part((uint64_t)G * G * b.WR * 4);
  cudaError_t e = b.mem.alloc(total, s);
  if (e != cudaSuccess) return build_fail(e, "alloc");
  char* mem = b.mem.as<char>();
  b.node = reinterpret_cast<uint64_t*>(mem + node_at);
  b.full = reinterpret_cast<uint64_t*>(mem + full_at);
  b.node_pre = reinterpret_cast<uint32_t*>(mem + np_at);
  b.leaf_pre = reinterpret_cast<uint32_t*>(mem + lp_at);
  uint16_t* leaves = reinterpret_cast<uint16_t*>(mem + lc_at);
  uint32_t* sums = reinterpret_cast<uint32_t*>(mem + sums_at);
  uint32_t* totals = reinterpret_cast<uint32_t*>(mem + tot_at);
  b.S = reinterpret_cast<uint32_t*>(mem + S_at);
  // the first words: levels 0 and 1 are written bytewise
  const size_t head = (b.nwords < 2u ? b.nwords : 2u) * 8u;
  if ((e = cudaMemsetAsync(b.node, 0, head, s)) != cudaSuccess ||
      (e = cudaMemsetAsync(b.full, 0, head, s)) != cudaSuccess)
    return build_fail(e, "clear");
  // (a view into a larger array need not be aligned for the 16-byte loads)
  if (G >= 128 && (reinterpret_cast<uintptr_t>(density) & 15u) == 0)
    solid_bits_v4_kernel<<<grid_for((uint64_t)G * G * b.WR * 8), 256, 0, s>>>(b.g, b.WR, b.S);
  else
    solid_bits_kernel<<<grid_for((uint64_t)G * G * b.WR * 32 / 4), 256, 0, s>>>(b.g, b.WR, b.S);
  classify_kernel<<<rows_blocks(b), 256, 0, s>>>(b.S, G, (int)b.WR, b.node + b.bottom,
                                                 b.full + b.bottom, leaves);
  // levels above, the large ones a launch each
  uint32_t at = b.bottom;
  int k = depth - 2;
  for (; k >= 0 && level_words(k + 1) > 8192u; --k) {
    const uint32_t words = level_words(k + 1), to = at - level_words(k);
    fold_kernel<<<(words + 255) / 256, 256, 0, s>>>(
        b.node + at, b.full + at, words, reinterpret_cast<uint8_t*>(b.node + to),
        reinterpret_cast<uint8_t*>(b.full + to));
    at = to;
  }
  if (k >= 0) fold_top_kernel<<<1, 1024, 0, s>>>(b.node, b.full, k);
  chunk_sums_kernel<<<nchunks + lchunks, 256, 0, s>>>(b.node, b.nwords, nchunks, leaves, lwords,
                                                      sums);
  chunk_scan_kernel<<<2, 1024, 0, s>>>(sums, nchunks, lchunks, totals);
  prefix_kernel<<<nchunks + lchunks, 256, 0, s>>>(b.node, b.nwords, nchunks, leaves, lwords, sums,
                                                  b.node_pre, b.leaf_pre);
  if ((e = cudaMemcpyAsync(totals + 2, b.full, 4, cudaMemcpyDeviceToDevice, s)) != cudaSuccess)
    return build_fail(e, "totals");
  uint32_t ht[3] = {};
  if ((e = cudaGetLastError()) != cudaSuccess ||
      (e = cudaMemcpyAsync(ht, totals, sizeof(ht), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
      (e = cudaStreamSynchronize(s)) != cudaSuccess)
    return build_fail(e, "totals");
  if (ht[0] == 0) {  // no surface voxel: the root is full or empty
    b.root = (ht[2] & 1u) ? YV_FULL_NODE : YV_EMPTY_NODE;
    return YV_OK;
  }
  if (ht[0] > YV_MAX_DEVICE_NODES) {
    set_last_error("dense SVO build: more than 2^29 nodes");
    return YV_ERR_UNSUPPORTED;
  }
  b.nn = ht[0];
  b.na = ht[1];
  b.root = 0;
  return YV_OK;
}

// Writes the nodes and leaves of a counted tree that has any.
template <bool kHost>
cudaError_t emit_dense(const SvoBuild& b, const BuildOut& out, cudaStream_t s) {
  if (b.bottom)
    emit_nodes_kernel<kHost><<<(b.bottom + 31) / 32, 256, 0, s>>>(b.node, b.full, b.node_pre,
                                                                 b.bottom, out);
  emit_bottom_kernel<kHost><<<8u * rows_blocks(b), 32, 0, s>>>(
      b.g, b.S, (int)b.WR, b.node + b.bottom, b.node_pre + b.bottom, b.leaf_pre, out);
  return cudaGetLastError();
}

}  // namespace
}  // namespace yv

using namespace yv;

extern "C" {

yv_status yv_svo_build_dense(const float* density, const uint8_t* rgb, int32_t depth, float iso,
                             void* stream, yv_svo_host** out) {
  if (!out) return YV_ERR_INVALID_ARG;
  *out = nullptr;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  SvoBuild b;
  yv_status st = count_dense(density, rgb, depth, iso, s, b);
  if (st != YV_OK) return st;
  std::vector<yv_vox_node> nodes(b.nn);
  std::vector<yv_leaf_attr> attrs(b.na);
  if (b.nn) {
    DevBuf dn, da;
    cudaError_t e;
    if ((e = dn.alloc((size_t)b.nn * sizeof(yv_vox_node), s)) != cudaSuccess ||
        (e = da.alloc((size_t)b.na * sizeof(yv_leaf_attr), s)) != cudaSuccess)
      return build_fail(e, "alloc");
    BuildOut o{};
    o.nodes = dn.as<yv_vox_node>();
    o.attrs = da.as<yv_leaf_attr>();
    if ((e = emit_dense<true>(b, o, s)) != cudaSuccess) return build_fail(e, "emit");
    e = cudaMemcpyAsync(nodes.data(), o.nodes, (size_t)b.nn * sizeof(yv_vox_node),
                        cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && b.na)
      e = cudaMemcpyAsync(attrs.data(), o.attrs, (size_t)b.na * sizeof(yv_leaf_attr),
                          cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return build_fail(e, "download");
  }
  return yv_svo_from_arrays(out, nodes.data(), b.nn, b.root, attrs.data(), b.na);
}

yv_status yv_set_scene_dense(yv_renderer* r, const float* density, const uint8_t* rgb,
                             int32_t depth, float iso, void* stream) {
  if (!r) return YV_ERR_INVALID_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  SvoBuild b;
  yv_status st = count_dense(density, rgb, depth, iso, s, b);
  if (st != YV_OK) return st;
  // straight into the renderer's (reused) scene buffers
  BuildOut o{};
  void* rec = nullptr;
  st = renderer_scene_buffers(r, b.nn, b.na, &o.rec, &o.cold, &rec);
  if (st != YV_OK) return st;
  o.shade = static_cast<uint4*>(rec);
  cudaError_t e = b.nn ? emit_dense<false>(b, o, s) : cudaSuccess;
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return build_fail(e, "emit");
  renderer_commit_scene(r, b.nn, b.na, (b.root & 0x80000000u) ? YV_DW_NULL : 0u);
  return YV_OK;
}

}  // extern "C"
