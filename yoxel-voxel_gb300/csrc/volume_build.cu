// volume_build.cu - GPU build of the ntree brick volume from a dense lattice:
// RangeBuilder (ntree/ntree/ntree.h:11-63) over an (S+1)^3 lattice, the
// producer side of the brick path (the GPU brick-pool construction of
// reaction/voxtree/density.cu:30-284 and BrickPool::Update,
// reaction/voxtree/brickpool/BrickPool.cpp:21-62: mark, scan, pack).
//
// Same result as the host builder yv_volume_from_dense, bit for bit: brick
// cells whose 9^3 lattice (with the far-side apron) holds a nonzero density
// are occupied; an N = 4 grid tree over them, grid nodes and bricks numbered
// in breadth-first order (children c = x | y<<2 | z<<4), the root always a
// grid node; bricks copy their 9^3 lattice values and RGB (white without an
// rgb lattice); neighbour tables for the apron fold.
//
// Passes: a cell is marked from per-row cell bits (the lattice read once) ORed
// over its 9 x 9 rows, 64 cells to a mask per last-level node; one pass per
// level above gathers the masks of its nodes; top-down, the prefix sums of the
// masks' counts expand level l's breadth-first list into level l+1's, give
// every node its first child and write its refs (bricks are the last level's
// children); a last pass packs the bricks (optionally straight into a device
// pool format) with their masks, bitmap and neighbours.  The passes over the
// tree take their sizes from the device; the host reads the counts once,
// before it sizes the pool.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "brick_mask.cuh"
#include "dev_scan.cuh"
#include "yv_internal.h"
#include "yv_kernels.h"

namespace yv {
namespace {

constexpr int kVB = 8;  // brick cells per axis
constexpr int kVL = 9;  // lattice points per axis with the apron
constexpr int kVL3 = 729;

struct Lattice {
  const float* d;
  const uint8_t* rgb;
  uint64_t L;  // lattice points per axis (S + 1)
  int nb;      // brick cells per axis
};

__device__ __forceinline__ uint64_t lat(const Lattice& g, int x, int y, int z) {
  return ((uint64_t)z * g.L + (uint64_t)y) * g.L + (uint64_t)x;
}

// Cell and level sizes are powers of two: index splits use shifts.

// Mark, pass 1: per lattice row (y, z), one bit per brick cell cx: some
// point of x in [8 cx, 8 cx + 8] (the cell's 8 points and its far apron
// point) is nonzero.  One warp per row reads it in coalesced 32-point chunks
// (eight loads in flight); the ballot of chunk j holds the points of cells
// 4j..4j+3, and a cell's apron point is the first point of the next cell.
// R[(z L + y) NW + w], NW = max(1, nb / 32) words per row.
__global__ void mark_rows_kernel(Lattice g, uint32_t* R) {
  constexpr int kU = 8;
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t rows = g.L * g.L;
  const uint32_t NW = g.nb >= 32 ? (uint32_t)g.nb / 32u : 1u;
  const uint32_t chunks = (uint32_t)((g.L + 31) / 32);  // 4 nb / 32 + 1
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t row = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; row < rows;
       row += nwarps) {
    const float* p = g.d + row * g.L;
    uint32_t word = 0, prev = 0;  // cell bits being assembled, previous chunk's ballot
    for (uint32_t j0 = 0; j0 < chunks; j0 += kU) {
      float v[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const uint64_t x = (uint64_t)(j0 + u) * 32u + lane;
        v[u] = (j0 + u < chunks && x < g.L) ? __ldg(p + x) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const uint32_t j = j0 + (uint32_t)u;
        if (j >= chunks) break;
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, v[u] != 0.f);
        if (j > 0) {
          // cells 4(j-1)..4(j-1)+3: own bytes of the previous chunk, apron =
          // the first bit of the following byte (bit 0 of this chunk for
          // the last one).  Bit 8k of `own` = byte k nonzero; the four
          // bits 0, 8, 16, 24 are gathered into bits 24..27 by one multiply
          // (no carries: the partial products below bit 24 are distinct).
          uint32_t own = prev | (prev >> 4);
          own |= own >> 2;
          own |= own >> 1;
          const uint32_t ap = (prev >> 8) | ((m & 1u) << 24);
          const uint32_t c4 = (((own | ap) & 0x01010101u) * 0x01020408u) >> 24;
          const uint32_t cbase = 4u * (j - 1);  // first cell of the group
          if (cbase < (uint32_t)g.nb) {
            word |= c4 << (cbase & 31u);
            if ((cbase & 31u) == 28u || cbase + 4u >= (uint32_t)g.nb) {
              if (lane == 0) R[row * NW + (cbase >> 5)] = word;
              word = 0;
            }
          }
        }
        prev = m;
      }
    }
  }
}

// Mark, pass 1, flat form (lattice 16-byte aligned, 16 <= nb <= 256, so a
// warp's 128 points touch at most two rows): the rows
// in groups of 4 (4 L floats start on a 16-byte boundary, L = 8 nb + 1 being
// odd only shifts the rows inside a group), read as float4 by one warp per
// group, 128 points per warp load, the next loads under way.  A lane marks the
// cells of its 4 points (own cell x >> 3, apron cell x / 8 - 1 for x a
// non-zero multiple of 8) in a 32-bit window of cells of the warp's row; one
// warp OR reduction per row the load touches (at most 2), and lane 0 merges it
// into the group's row words in shared memory.  A bit past the last cell (its
// apron point) is dropped with the words or masked at the end.  Same R as
// mark_rows_kernel.  513^3: 155 us with per-point tests of row and cell, 138 us
// one load at a time, 122 us with 4 under way (128 with 2 or 8).
constexpr uint32_t kFlatMaxNW = 8;
constexpr uint32_t kFlatAhead = 4;  // loads a lane has under way

__global__ void mark_rows_flat_kernel(Lattice g, uint32_t* R) {
  __shared__ uint32_t acc_all[8][4][kFlatMaxNW];
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t(*acc)[kFlatMaxNW] = acc_all[(threadIdx.x >> 5) & 7u];
  const uint32_t L = (uint32_t)g.L;
  const uint32_t nb = (uint32_t)g.nb;
  const uint32_t NW = nb >= 32 ? nb / 32u : 1u;
  const uint64_t rows = g.L * g.L;
  const uint64_t groups = (rows + 3) / 4;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const float4* d4 = reinterpret_cast<const float4*>(g.d);
  for (uint64_t grp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; grp < groups;
       grp += nwarps) {
    const uint64_t left_rows = rows - grp * 4;
    const uint32_t nrows = left_rows < 4 ? (uint32_t)left_rows : 4u;
    const uint32_t nfl = nrows * L;             // floats of the group
    const uint32_t n4 = (nfl + 3) / 4;          // float4 loads (the last may run past)
    if (lane < 4 * kFlatMaxNW) acc[lane >> 3][lane & 7u] = 0u;
    __syncwarp();
    const float4* src = d4 + grp * (uint64_t)L;  // 4 L floats = L float4
    // row and x of the warp's first point, advanced by 128 points a step
    // (L > 128: at most one row boundary per step)
    uint32_t ra = 0, xs = 0;
    for (uint32_t f1 = 0; f1 < n4; f1 += 32u * kFlatAhead) {
      float4 ahead[kFlatAhead];
#pragma unroll
      for (uint32_t u = 0; u < kFlatAhead; ++u) {
        const uint32_t f = f1 + 32u * u + lane;
        ahead[u] = 4u * f + 3u < nfl ? __ldg(src + f) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (uint32_t u = 0; u < kFlatAhead; ++u) {
        const uint32_t f0 = f1 + 32u * u, f = f0 + lane;
        if (f0 >= n4) break;
        float4 v = ahead[u];
        if (4u * f + 3u >= nfl && f < n4) {
          // the group's (and the lattice's) last points: no read past them
          const float* s1 = reinterpret_cast<const float*>(src) + 4u * f;
          const uint32_t left = nfl - 4u * f;
          v.x = __ldg(s1);
          if (left > 1u) v.y = __ldg(s1 + 1);
          if (left > 2u) v.z = __ldg(s1 + 2);
        }
        // the lane's 4 points, the first `own` of them in row ra, the rest in
        // the next; shifted to their place among the 8 of their cell, bit 0 is
        // also the previous cell's apron, bit 8 the next cell's first point and
        // this one's apron.  Window bit 0: the cell before the warp's first
        // (row ra), cell -1 (the next row).
        const uint32_t nib = (v.x != 0.f ? 1u : 0u) | (v.y != 0.f ? 2u : 0u) |
                             (v.z != 0.f ? 4u : 0u) | (v.w != 0.f ? 8u : 0u);
        const uint32_t xl = xs + 4u * lane;
        const uint32_t own = xl >= L ? 0u : (L - xl < 4u ? L - xl : 4u);
        {
          const uint32_t q = (xs & 7u) + 4u * lane;
          const uint32_t p = (nib & ((1u << own) - 1u)) << (q & 7u);
          const uint32_t bits = (p & 1u) | ((p & 0x1FFu) ? 2u : 0u) | ((p >> 8) ? 4u : 0u);
          const uint32_t win = __reduce_or_sync(0xFFFFFFFFu, bits << (q >> 3));
          if (lane == 0 && win) {
            const uint32_t c = xs >> 3;
            const uint64_t sft = c ? (uint64_t)win << ((c - 1u) & 31u) : (uint64_t)(win >> 1);
            const uint32_t w = c ? (c - 1u) >> 5 : 0u;
            if (w < NW) acc[ra][w] |= (uint32_t)sft;
            if (w + 1 < NW) acc[ra][w + 1] |= (uint32_t)(sft >> 32);
          }
        }
        if (xs + 128u > L) {  // the whole warp
          const uint32_t q = xl >= L ? xl - L : 0u;
          const uint32_t p = (nib >> own) << (q & 7u);
          const uint32_t bits = (p & 1u) | ((p & 0x1FFu) ? 2u : 0u) | ((p >> 8) ? 4u : 0u);
          const uint32_t win = __reduce_or_sync(0xFFFFFFFFu, bits << (q >> 3));
          if (lane == 0 && win && ra + 1u < nrows) acc[ra + 1u][0] |= win >> 1;
        }
        xs += 128u;
        if (xs >= L) {
          xs -= L;
          ++ra;
        }
      }
    }
    __syncwarp();
    if (lane < nrows * NW) {
      const uint32_t r = lane / NW, w = lane % NW;
      R[(grp * 4 + r) * NW + w] = acc[r][w] & (nb >= 32 ? 0xFFFFFFFFu : ((1u << nb) - 1u));
    }
    __syncwarp();
  }
}

// Mark, pass 2: a cell is occupied when its bit is set in any of the 9 x 9
// rows y in [8 cy, 8 cy + 8], z in [8 cz, 8 cz + 8].  One warp per row word and
// 4x4 square of (cy, cz): lane j and j + 16 OR the lower and upper rows of
// square cell j, then the nibbles of the 16 lanes make the 64-cell mask (bit
// x | y<<2 | z<<4) of each last-level node of the word.
// node_count += nodes with a cell, cell_count += cells.
__global__ void __launch_bounds__(256) mark_nodes_kernel(Lattice g, const uint32_t* R,
                                                         uint64_t* mask, uint32_t* node_count,
                                                         uint32_t* cell_count) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t NW = g.nb >= 32 ? (uint32_t)g.nb / 32u : 1u;
  const uint32_t n = (uint32_t)g.nb / 4u;  // nodes per axis
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (warp >= NW * n * n) return;
  const uint32_t w = warp % NW, gy = (warp / NW) % n, gz = warp / (NW * n);
  const uint32_t y = lane & 3u, z = (lane >> 2) & 3u;
  const uint64_t cy = 4u * gy + y, cz = 4u * gz + z;
  const int z0 = lane < 16u ? 0 : 5, z1 = lane < 16u ? 5 : 9;
  uint32_t acc = 0;
  for (int dz = z0; dz < z1; ++dz) {
    const uint32_t* p = R + ((8u * cz + (uint64_t)dz) * g.L + 8u * cy) * NW + w;
#pragma unroll
    for (int dy = 0; dy < 9; ++dy) acc |= __ldg(p + (uint32_t)dy * NW);
  }
  acc |= __shfl_xor_sync(0xFFFFFFFFu, acc, 16);
  const uint32_t nn = n < 8u ? n : 8u;
  uint32_t lo = 0, hi = 0;  // lane k: the mask of node k of the word
  for (uint32_t k = 0; k < nn; ++k) {
    const uint32_t nib = ((acc >> (4u * k)) & 15u) << (4u * y + 16u * (z & 1u));
    const uint32_t l = __reduce_or_sync(0xFFFFFFFFu, z < 2u ? nib : 0u);
    const uint32_t h = __reduce_or_sync(0xFFFFFFFFu, z < 2u ? 0u : nib);
    if (lane == k) {
      lo = l;
      hi = h;
    }
  }
  if (lane < nn)
    mask[((uint64_t)gz * n + gy) * n + 8u * w + lane] = (uint64_t)lo | ((uint64_t)hi << 32);
  const uint32_t cells = __reduce_add_sync(0xFFFFFFFFu, __popc(lo) + __popc(hi));
  const uint32_t nodes = __popc(__ballot_sync(0xFFFFFFFFu, (lo | hi) != 0u));
  if (lane == 0 && cells) {
    atomicAdd(cell_count, cells);
    atomicAdd(node_count, nodes);
  }
}

// Index of child c (x | y<<2 | z<<4) of node p of a level with n = 2^s
// nodes per axis, in the level below (4n per axis).
__device__ __forceinline__ uint32_t child64(uint32_t p, uint32_t n, uint32_t c) {
  const int s = __ffs(n) - 1;
  const uint32_t x = p & (n - 1u), y = (p >> s) & (n - 1u), z = p >> (2 * s);
  return (4 * x + (c & 3u)) + ((4 * y + ((c >> 2) & 3u)) << (s + 2)) +
         ((4 * z + (c >> 4)) << (2 * s + 4));
}

// Masks of level l (n per axis) from level l+1's (4n per axis), a warp per
// node; count += nodes with a child.
__global__ void __launch_bounds__(256) fold_masks_kernel(const uint64_t* child, uint32_t n,
                                                         uint64_t* mask, uint32_t* count) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (p >= n * n * n) return;
  const uint32_t lo = __ballot_sync(0xFFFFFFFFu, child[child64(p, n, lane)] != 0ull);
  const uint32_t hi = __ballot_sync(0xFFFFFFFFu, child[child64(p, n, lane + 32u)] != 0ull);
  if (lane == 0) {
    mask[p] = (uint64_t)lo | ((uint64_t)hi << 32);
    if (lo | hi) atomicAdd(count, 1u);
  }
}

// Nodes of level l's breadth-first list per block of the two kernels below.
constexpr uint32_t kListChunk = 256;

// counts: occupied nodes of each level ([0] unused: the root is always
// there).  Length of level l's list.
__device__ __forceinline__ uint32_t list_len(const uint32_t* counts, int l) {
  return l == 0 ? 1u : counts[l];
}

// Children per chunk of level l's list.
__global__ void __launch_bounds__(kListChunk) child_sums_kernel(const uint32_t* counts, int l,
                                                                const uint32_t* list,
                                                                const uint64_t* mask,
                                                                uint32_t* sums) {
  const uint32_t m = list_len(counts, l), i = blockIdx.x * kListChunk + threadIdx.x;
  if (blockIdx.x * kListChunk >= m) return;
  __shared__ uint32_t tot;
  if (threadIdx.x == 0) tot = 0;
  __syncthreads();
  uint32_t c = i < m ? (uint32_t)__popcll(mask[list[i]]) : 0u;
  c = __reduce_add_sync(0xFFFFFFFFu, c);
  if ((threadIdx.x & 31u) == 0 && c) atomicAdd(&tot, c);
  __syncthreads();
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// Level l's nodes: their place in the next list (the sums of the chunks
// before, then a scan of the chunk), the next list itself and the refs -
// occupied children are grid nodes or, at the last level, bricks
// (0x40000000 | rank; map[cell] = rank).  A warp per node writes its 64 refs.
// sums: children per chunk (null: one chunk holds the list).
__global__ void __launch_bounds__(kListChunk)
    expand_kernel64(const uint32_t* counts, int l, bool last, uint32_t n, const uint32_t* list,
                    const uint64_t* mask, const uint32_t* sums, uint32_t* next, uint32_t* grids,
                    int32_t* map) {
  __shared__ uint64_t s_mask[kListChunk];
  __shared__ uint32_t s_off[kListChunk], s_node[kListChunk], s_warp[kListChunk / 32], s_base;
  const uint32_t m = list_len(counts, l), i0 = blockIdx.x * kListChunk;
  if (i0 >= m) return;
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  if (t == 0) s_base = 0;
  __syncthreads();
  if (sums) {
    uint32_t b = 0;
    for (uint32_t k = t; k < blockIdx.x; k += kListChunk) b += sums[k];
    b = __reduce_add_sync(0xFFFFFFFFu, b);
    if (lane == 0 && b) atomicAdd(&s_base, b);
  }
  const uint32_t here = m - i0 < kListChunk ? m - i0 : kListChunk;
  const uint32_t p = t < here ? list[i0 + t] : 0u;
  const uint64_t mk = t < here ? mask[p] : 0ull;
  uint32_t inc = (uint32_t)__popcll(mk);
  const uint32_t own = inc;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
    if (lane >= (uint32_t)o) inc += u;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  uint32_t off = s_base + inc - own;
  for (uint32_t w = 0; w < warp; ++w) off += s_warp[w];
  s_mask[t] = mk;
  s_off[t] = off;
  s_node[t] = p;
  __syncthreads();
  uint32_t node_base = 0, child_base = 1;  // grid nodes before this level, before the next
  for (int k = 0; k < l; ++k) {
    node_base = child_base;
    child_base += counts[k + 1];
  }
  for (uint32_t j = warp; j < here; j += kListChunk / 32) {
    const uint64_t bits = s_mask[j];
    const uint32_t o = s_off[j], q = s_node[j];
    uint32_t* g = grids + (size_t)(node_base + i0 + j) * 64;
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
      const uint32_t c = lane + 32u * h;
      uint32_t ref = 0x80000000u;
      if ((bits >> c) & 1ull) {
        const uint32_t rank = o + (uint32_t)__popcll(bits & ((1ull << c) - 1ull));
        const uint32_t ch = child64(q, n, c);
        next[rank] = ch;
        ref = last ? (0x40000000u | rank) : child_base + rank;
        if (last && map) map[ch] = (int32_t)rank;
      }
      g[c] = ref;
    }
  }
}

__device__ __forceinline__ uint16_t f16_saturating(float f) {
  if (f != f) return 0;  // NaN -> 0, as the host upload
  uint16_t u = __half_as_ushort(__float2half_rn(f));
  if ((u & 0x7FFFu) == 0x7C00u) u = (uint16_t)((u & 0x8000u) | 0x7BFFu);
  return u;
}

// RGB of lattice point i (R in the low byte) from two aligned words, or byte by
// byte at the array's end and where the array is not 4-byte aligned (words =
// the whole words of the array, 0 then).
__device__ __forceinline__ uint32_t load_rgb(const uint8_t* rgb, uint64_t i, uint64_t words) {
  const uint64_t b = 3u * i, w = b >> 2;
  if (w + 1 < words) {
    const uint32_t* p = reinterpret_cast<const uint32_t*>(rgb) + w;
    return __funnelshift_r(__ldg(p), __ldg(p + 1), ((uint32_t)b & 3u) * 8u) & 0xFFFFFFu;
  }
  return (uint32_t)rgb[b] | ((uint32_t)rgb[b + 1] << 8) | ((uint32_t)rgb[b + 2] << 16);
}

// Apron neighbours of a brick (index m-1 for the offset m = dx | dy<<1 |
// dz<<2), lanes 0..6 the upper and 8..14 the lower ones.
__device__ __forceinline__ void write_neighbors(const int32_t* map, int nb, uint32_t b, int x,
                                                int y, int z, uint32_t lane, int32_t* up,
                                                int32_t* dn) {
  const int m = (int)(lane & 7u) + 1;
  if (m > 7 || lane > 14u) return;
  const int s = lane < 8u ? 1 : -1;
  const int ux = x + s * (m & 1), uy = y + s * ((m >> 1) & 1), uz = z + s * (m >> 2);
  const bool in = ux >= 0 && uy >= 0 && uz >= 0 && ux < nb && uy < nb && uz < nb;
  const int32_t v = in ? map[((size_t)uz * nb + uy) * nb + ux] : -1;
  (lane < 8u ? up : dn)[7 * (size_t)b + (size_t)(m - 1)] = v;
}

// Pack: one warp per brick, its 729 lattice values (and RGB).  kFormat < 0:
// fp32 density + uint8 RGB (host container layout); else a device pool
// format (YV_PRECISION_*), written to d_out / a_out.
// The lattice offset of each of the 729 points from a brick's first is one
// table in shared memory; loads of 8 points are issued before any is used.
// 513^3 lattice with colours, 74 k bricks, 8-byte format: 566 us with the
// offsets and three byte loads worked out per point, 283 us so, 235 us with
// registers for 6 blocks an SM (4 without the bound; 8 spill: 270 us): bound
// by the latency of its loads.
// Device pools (kFormat >= 0): mask is the cell occupancy mask of the march
// (16 words per brick, cell_mask_word) of the stored densities; bits
// (optional, zeroed before) the brick bitmap, bit (ci & 31) of word ci >> 5
// set for the cell ci = (cz nb + cy) nb + cx of every brick; up / dn the apron
// neighbours.  Host container: cell_xyz.
template <int kFormat>
__global__ void __launch_bounds__(256, 6)
    pack_bricks_kernel(Lattice g, const uint32_t* cells, uint32_t nbricks, uint64_t rgb_words,
                       float* dens, uint8_t* rgb, void* d_out, void* a_out, int32_t* cell_xyz,
                       const int32_t* map, int32_t* up, int32_t* dn, uint32_t* mask,
                       uint32_t* bits) {
  __shared__ uint32_t nzbits[8][24];
  __shared__ uint32_t offs[kVL3 + 7];
  const uint32_t L = (uint32_t)g.L;
  for (uint32_t k = threadIdx.x; k < kVL3; k += blockDim.x)
    offs[k] = k % kVL + ((k / kVL) % kVL) * L + (k / (kVL * kVL)) * L * L;
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t* nz = nzbits[threadIdx.x >> 5];
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const int nbs = __ffs(g.nb) - 1;
  constexpr bool kHalf = kFormat == YV_PRECISION_F16 || kFormat == YV_PRECISION_F16_PACKED;
  for (uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < nbricks; b += nwarps) {
    const uint32_t c = cells[b];
    const int cx = (int)(c & (uint32_t)(g.nb - 1)), cy = (int)((c >> nbs) & (uint32_t)(g.nb - 1)),
              cz = (int)(c >> (2 * nbs));
    if (kFormat < 0) {
      if (lane == 0) {
        cell_xyz[3 * (size_t)b] = cx;
        cell_xyz[3 * (size_t)b + 1] = cy;
        cell_xyz[3 * (size_t)b + 2] = cz;
      }
    } else {
      write_neighbors(map, g.nb, b, cx, cy, cz, lane, up, dn);
      // the linear cell index is c itself
      if (lane == 31 && bits) atomicOr(bits + (c >> 5), 1u << (c & 31u));
    }
    const uint64_t first = lat(g, cx * kVB, cy * kVB, cz * kVB);
    const float* src = g.d + first;
    const size_t o0 = (size_t)b * kVL3;
    for (uint32_t q0 = 0; q0 < 24u; q0 += 8u) {
      float pv[8];
      uint32_t pc[8];
#pragma unroll
      for (uint32_t u = 0; u < 8u; ++u) {
        const uint32_t k = lane + 32u * (q0 + u);
        const bool in = k < (uint32_t)kVL3;
        const uint32_t o = in ? offs[k] : 0u;
        pv[u] = in ? __ldg(src + o) : 0.f;
        pc[u] = g.rgb ? load_rgb(g.rgb, first + o, rgb_words) : 0xFFFFFFu;
      }
#pragma unroll
      for (uint32_t u = 0; u < 8u; ++u) {
        const uint32_t k = lane + 32u * (q0 + u);
        const float v = pv[u];
        const uint32_t r = pc[u] & 0xFFu, gg = (pc[u] >> 8) & 0xFFu, bb = pc[u] >> 16;
        const uint32_t h = kHalf ? (uint32_t)f16_saturating(v) : 0u;
        if (kFormat >= 0) {
          // the non-zero points as stored (the fp16 formats round small
          // values to 0); zero beyond the 729 points
          const bool nzv = kHalf ? (h & 0x7FFFu) != 0u : v != 0.f;
          const uint32_t bal = __ballot_sync(0xFFFFFFFFu, nzv);
          if (lane == 0) nz[q0 + u] = bal;
        }
        if (k < (uint32_t)kVL3) {
          const size_t o = o0 + k;
          if (kFormat < 0) {
            dens[o] = v;
            rgb[3 * o] = (uint8_t)r;
            rgb[3 * o + 1] = (uint8_t)gg;
            rgb[3 * o + 2] = (uint8_t)bb;
          } else if (kFormat == YV_PRECISION_F16) {
            static_cast<uint16_t*>(d_out)[o] = (uint16_t)h;
            static_cast<uint32_t*>(a_out)[o] = pc[u] | 0xFF000000u;
          } else if (kFormat == YV_PRECISION_F32) {
            static_cast<float*>(d_out)[o] = v;
            float* a = static_cast<float*>(a_out) + 3 * o;
            a[0] = __fmul_rn((float)r, 1.0f / 255.0f);
            a[1] = __fmul_rn((float)gg, 1.0f / 255.0f);
            a[2] = __fmul_rn((float)bb, 1.0f / 255.0f);
          } else if (kFormat == YV_PRECISION_F32_PACKED) {
            static_cast<float4*>(a_out)[o] =
                make_float4(__fmul_rn((float)r, 1.0f / 255.0f), __fmul_rn((float)gg, 1.0f / 255.0f),
                            __fmul_rn((float)bb, 1.0f / 255.0f), v);
          } else {
            static_cast<uint2*>(a_out)[o] = make_uint2(h | (pc[u] << 16), bb);
          }
        }
      }
    }
    if (kFormat >= 0) {
      __syncwarp();
      if (lane < 16u) mask[(size_t)b * 16u + lane] = cell_mask_word(nz, lane);
      __syncwarp();
    }
  }
}

// Whole aligned words of the lattice's colours, 0 where the words cannot be
// read (unaligned).
uint64_t rgb_words(const Lattice& g) {
  if (!g.rgb || (reinterpret_cast<uintptr_t>(g.rgb) & 3u)) return 0;
  return 3u * g.L * g.L * g.L / 4u;
}

yv_status vbuild_fail(cudaError_t e, const char* what) {
  set_last_error(std::string("dense volume build: ") + what + ": " + cudaGetErrorString(e));
  cudaGetLastError();
  return e == cudaErrorMemoryAllocation ? YV_ERR_OUT_OF_MEMORY : YV_ERR_CUDA;
}

// Tree of a dense lattice on the device: grid refs (ngrids x 64), the
// breadth-first brick cells and the brick of every cell (-1: none), in one
// scratch allocation sized for a full tree.
struct VolumeTree {
  DevBuf mem;
  uint32_t* grids = nullptr;
  uint32_t* cells = nullptr;
  int32_t* map = nullptr;
  uint32_t ngrids = 0, nbricks = 0;
};

yv_status build_volume_tree(const Lattice& g, int levels, cudaStream_t s, VolumeTree& t) {
  const uint64_t NW = g.nb >= 32 ? (uint64_t)g.nb / 32 : 1;
  const uint64_t cells = (uint64_t)g.nb * g.nb * g.nb;
  // the parts of the scratch, 256-byte aligned: node masks and lists per
  // level, sums of the largest list, grid refs, cell map, row bits, counts
  uint64_t total = 0, max_grids = 0;
  auto part = [&](uint64_t bytes) {
    const uint64_t at = total;
    total += (bytes + 255u) & ~255ull;
    return at;
  };
  uint64_t mask_at[5], list_at[6];
  for (int l = 0; l < levels; ++l) {
    mask_at[l] = part((1ull << (6 * l)) * 8);
    max_grids += 1ull << (6 * l);
  }
  for (int l = 0; l <= levels; ++l) list_at[l] = part((1ull << (6 * l)) * 4);
  const uint64_t sums_at = part(((1ull << (6 * (levels - 1))) / kListChunk + 1) * 4);
  const uint64_t grids_at = part(max_grids * 256);
  const uint64_t map_at = part(cells * 4);
  const uint64_t rows_at = part(g.L * g.L * NW * 4);
  const uint64_t counts_at = part(256);
  cudaError_t e = t.mem.alloc(total, s);
  if (e != cudaSuccess) return vbuild_fail(e, "alloc");
  char* mem = t.mem.as<char>();
  auto mask = [&](int l) { return reinterpret_cast<uint64_t*>(mem + mask_at[l]); };
  auto list = [&](int l) { return reinterpret_cast<uint32_t*>(mem + list_at[l]); };
  uint32_t* sums = reinterpret_cast<uint32_t*>(mem + sums_at);
  uint32_t* rows = reinterpret_cast<uint32_t*>(mem + rows_at);
  uint32_t* counts = reinterpret_cast<uint32_t*>(mem + counts_at);
  t.grids = reinterpret_cast<uint32_t*>(mem + grids_at);
  t.cells = list(levels);
  t.map = reinterpret_cast<int32_t*>(mem + map_at);
  if ((e = cudaMemsetAsync(counts, 0, 256, s)) != cudaSuccess ||
      (e = cudaMemsetAsync(list(0), 0, 4, s)) != cudaSuccess ||
      (e = cudaMemsetAsync(t.map, 0xFF, cells * 4, s)) != cudaSuccess)
    return vbuild_fail(e, "clear");
  if (g.nb >= 16 && NW <= kFlatMaxNW && (reinterpret_cast<uintptr_t>(g.d) & 15u) == 0)
    mark_rows_flat_kernel<<<grid_for((g.L * g.L + 3) / 4 * 32), 256, 0, s>>>(g, rows);
  else
    mark_rows_kernel<<<grid_for(g.L * g.L * 32), 256, 0, s>>>(g, rows);
  // a warp per word and 4x4 square of cells
  const uint64_t n4 = (uint64_t)g.nb / 4;
  mark_nodes_kernel<<<(unsigned)((NW * n4 * n4 + 7) / 8), 256, 0, s>>>(
      g, rows, mask(levels - 1), counts + (levels > 1 ? levels - 1 : 8), counts + levels);
  for (int l = levels - 2; l >= 0; --l) {
    const uint32_t n = 1u << (2 * l);
    fold_masks_kernel<<<(unsigned)(((uint64_t)n * n * n + 7) / 8), 256, 0, s>>>(
        mask(l + 1), n, mask(l), counts + (l > 0 ? l : 8));  // [8]: not read
  }
  for (int l = 0; l < levels; ++l) {
    const uint32_t chunks = (uint32_t)(((1ull << (6 * l)) + kListChunk - 1) / kListChunk);
    if (chunks > 1)
      child_sums_kernel<<<chunks, kListChunk, 0, s>>>(counts, l, list(l), mask(l), sums);
    expand_kernel64<<<chunks, kListChunk, 0, s>>>(counts, l, l == levels - 1, 1u << (2 * l),
                                                  list(l), mask(l), chunks > 1 ? sums : nullptr,
                                                  list(l + 1), t.grids, t.map);
  }
  uint32_t hc[8] = {};
  if ((e = cudaGetLastError()) != cudaSuccess ||
      (e = cudaMemcpyAsync(hc, counts, sizeof(hc), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
      (e = cudaStreamSynchronize(s)) != cudaSuccess)
    return vbuild_fail(e, "tree");
  // grid nodes: the root and the occupied nodes of levels 1..levels-1
  t.ngrids = 1;
  for (int l = 1; l < levels; ++l) t.ngrids += hc[l];
  t.nbricks = hc[levels];
  return YV_OK;
}

bool lattice_args(const float* density, int levels, Lattice* g, const uint8_t* rgb) {
  if (!density || levels < 1 || levels > 4) return false;
  g->d = density;
  g->rgb = rgb;
  g->nb = 1 << (2 * levels);
  g->L = (uint64_t)g->nb * kVB + 1;
  return true;
}

}  // namespace
}  // namespace yv

using namespace yv;

extern "C" {

yv_status yv_volume_build_dense(const float* density, const uint8_t* rgb, int32_t levels,
                                void* stream, yv_volume_host** out) {
  if (!out) return YV_ERR_INVALID_ARG;
  *out = nullptr;
  Lattice g;
  if (!lattice_args(density, levels, &g, rgb)) return YV_ERR_INVALID_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  VolumeTree t;
  yv_status st = build_volume_tree(g, levels, s, t);
  if (st != YV_OK) return st;
  const size_t n = (size_t)t.nbricks * kVL3;
  DevBuf dens, col, cxyz;
  cudaError_t e;
  if ((e = dens.alloc(n * 4, s)) != cudaSuccess || (e = col.alloc(n * 3, s)) != cudaSuccess ||
      (e = cxyz.alloc((size_t)t.nbricks * 12, s)) != cudaSuccess)
    return vbuild_fail(e, "alloc");
  if (t.nbricks)
    pack_bricks_kernel<-1><<<grid_for((uint64_t)t.nbricks * 32), 256, 0, s>>>(
        g, t.cells, t.nbricks, rgb_words(g), dens.as<float>(), col.as<uint8_t>(), nullptr,
        nullptr, cxyz.as<int32_t>(), nullptr, nullptr, nullptr, nullptr, nullptr);
  if ((e = cudaGetLastError()) != cudaSuccess) return vbuild_fail(e, "pack");
  std::vector<uint32_t> grids((size_t)t.ngrids * 64);
  std::vector<float> hd(n);
  std::vector<uint8_t> hc(n * 3);
  std::vector<int32_t> hcell((size_t)t.nbricks * 3);
  if ((e = cudaMemcpyAsync(grids.data(), t.grids, grids.size() * 4, cudaMemcpyDeviceToHost,
                           s)) != cudaSuccess ||
      (n && (e = cudaMemcpyAsync(hd.data(), dens.p, n * 4, cudaMemcpyDeviceToHost, s)) !=
                cudaSuccess) ||
      (n && (e = cudaMemcpyAsync(hc.data(), col.p, n * 3, cudaMemcpyDeviceToHost, s)) !=
                cudaSuccess) ||
      (t.nbricks && (e = cudaMemcpyAsync(hcell.data(), cxyz.p, hcell.size() * 4,
                                         cudaMemcpyDeviceToHost, s)) != cudaSuccess) ||
      (e = cudaStreamSynchronize(s)) != cudaSuccess)
    return vbuild_fail(e, "download");
  return volume_host_from_parts(levels, std::move(grids), std::move(hd), std::move(hc),
                                std::move(hcell), out);
}

}  // extern "C"

namespace yv {
namespace {

// Builds the device pool from a lattice into `into` (reusing its arrays
// where they are large enough) or into a new volume (*out).
yv_status upload_dense(const float* density, const uint8_t* rgb, int32_t levels,
                       int32_t precision, cudaStream_t s, yv_volume_gpu* into,
                       yv_volume_gpu** out) {
  Lattice g;
  if (!lattice_args(density, levels, &g, rgb) || precision < YV_PRECISION_F16 ||
      precision > YV_PRECISION_F16_PACKED)
    return YV_ERR_INVALID_ARG;
  VolumeTree t;
  yv_status st = build_volume_tree(g, levels, s, t);
  if (st == YV_OK) st = pool_points_fit(t.nbricks);
  if (st != YV_OK) return st;
  const size_t n = (size_t)t.nbricks * kVL3;
  size_t dbytes = 0, abytes = 0;
  switch (precision) {
    case YV_PRECISION_F16: dbytes = n * 2; abytes = n * 4; break;
    case YV_PRECISION_F32: dbytes = n * 4; abytes = n * 12; break;
    case YV_PRECISION_F32_PACKED: abytes = n * 16; break;
    default: abytes = n * 8; break;
  }
  // the device pool (owned by the yv_volume_gpu): grids, density, albedo,
  // neighbours up / down
  const size_t bytes[5] = {(size_t)t.ngrids * 256, dbytes, abytes, (size_t)t.nbricks * 28,
                           (size_t)t.nbricks * 28};
  void* fresh[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  void** mem = fresh;
  size_t* cap = nullptr;
  yv_volume_device* desc = nullptr;
  if (into) volume_gpu_arrays(into, &mem, &cap, &desc);
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < 5 && e == cudaSuccess; ++i) {
    if (!bytes[i] || (cap && cap[i] >= bytes[i])) continue;
    if (cap) {
      // grow: the old array may still be read by queued work on `s`
      e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) break;
      cudaFree(mem[i]);
      mem[i] = nullptr;
      cap[i] = 0;
    }
    e = cudaMalloc(&mem[i], bytes[i]);
    if (e == cudaSuccess && cap) cap[i] = bytes[i];
  }
  // the acceleration arrays: the cell occupancy mask (written by the pack
  // kernel), then the brick bitmap
  uint32_t *mask = nullptr, *bits = nullptr;
  if (e == cudaSuccess && t.nbricks) {
    if (into) {
      const yv_status mst = volume_gpu_accel_buffer(into, t.nbricks, levels, s, &mask, &bits);
      if (mst != YV_OK) return mst;
    } else {
      e = cudaMalloc(&mask, volume_accel_bytes(t.nbricks, levels));
      if (e == cudaSuccess && levels <= 4) bits = mask + (size_t)t.nbricks * 16u;
    }
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(mem[0], t.grids, bytes[0], cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess && bits)
    e = cudaMemsetAsync(bits, 0, (size_t)YV_BRICK_BITS_WORDS(levels) * 4u, s);
  if (e == cudaSuccess && t.nbricks) {
    auto kern = precision == YV_PRECISION_F16          ? pack_bricks_kernel<YV_PRECISION_F16>
                : precision == YV_PRECISION_F32        ? pack_bricks_kernel<YV_PRECISION_F32>
                : precision == YV_PRECISION_F32_PACKED
                    ? pack_bricks_kernel<YV_PRECISION_F32_PACKED>
                    : pack_bricks_kernel<YV_PRECISION_F16_PACKED>;
    kern<<<grid_for((uint64_t)t.nbricks * 32), 256, 0, s>>>(
        g, t.cells, t.nbricks, rgb_words(g), nullptr, nullptr, mem[1], mem[2], nullptr, t.map,
        static_cast<int32_t*>(mem[3]), static_cast<int32_t*>(mem[4]), mask, bits);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    if (!into) {
      for (void* p : fresh) cudaFree(p);
      cudaFree(mask);
    }
    return vbuild_fail(e, "device pool");
  }
  yv_volume_device d;
  d.grids = static_cast<const uint32_t*>(mem[0]);
  d.ngrids = t.ngrids;
  d.levels = levels;
  d.density = mem[1];
  d.albedo = mem[2];
  d.nbricks = t.nbricks;
  d.precision = precision;
  d.nbr_up = static_cast<const int32_t*>(mem[3]);
  d.nbr_dn = static_cast<const int32_t*>(mem[4]);
  d.cell_mask = mask;
  d.brick_bits = bits;
  if (into) {
    *desc = d;
    return YV_OK;
  }
  // a new volume: its buffers are complete once the stream gets here
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) {
    for (void* p : fresh) cudaFree(p);
    cudaFree(mask);
    return vbuild_fail(e, "device pool");
  }
  return volume_gpu_from_device(fresh, bytes, d, out, mask);
}

}  // namespace
}  // namespace yv

extern "C" {

yv_status yv_volume_upload_dense(const float* density, const uint8_t* rgb, int32_t levels,
                                 int32_t precision, void* stream, yv_volume_gpu** out) {
  if (!out) return YV_ERR_INVALID_ARG;
  *out = nullptr;
  return upload_dense(density, rgb, levels, precision, static_cast<cudaStream_t>(stream),
                      nullptr, out);
}

yv_status yv_volume_rebuild_dense(yv_volume_gpu* vol, const float* density, const uint8_t* rgb,
                                  int32_t levels, void* stream) {
  if (!vol) return YV_ERR_INVALID_ARG;
  yv_volume_device d;
  yv_status st = yv_volume_gpu_desc(vol, &d);
  if (st != YV_OK) return st;
  return upload_dense(density, rgb, levels, d.precision, static_cast<cudaStream_t>(stream), vol,
                      nullptr);
}

}  // extern "C"
