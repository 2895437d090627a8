// brick_mask.cuh - cell occupancy mask of a brick from the bits of its lattice
// points, shared by the kernels that pack a pool (volume_build.cu,
// brick_kernels.cu).
#pragma once
#include <cstdint>

namespace yv {
namespace {

// Bits of the 9 lattice points from offset `off` of a brick's 729-bit map.
__device__ __forceinline__ uint32_t lattice_row9(const uint32_t* bits, int off) {
  const int w = off >> 5, sh = off & 31;
  uint32_t v = bits[w] >> sh;
  if (sh > 23) v |= bits[w + 1] << (32 - sh);
  return v & 0x1FFu;
}

// Word w (0..15) of a brick's cell occupancy mask from the 729-bit map of its
// lattice points (24 words, bits past 729 zero): bit (y & 3) * 8 + x set
// where a corner of trilinear cell (x, y, z) is set, w = z * 2 + (y >> 2).
__device__ __forceinline__ uint32_t cell_mask_word(const uint32_t* nz, uint32_t w) {
  const int z = (int)(w >> 1), y0 = (int)(w & 1u) * 4;
  uint32_t word = 0;
  for (int yy = 0; yy < 4; ++yy) {
    uint32_t rows = 0;
    for (int dz = 0; dz < 2; ++dz)
      for (int dy = 0; dy < 2; ++dy) {
        const uint32_t r9 = lattice_row9(nz, (z + dz) * 81 + (y0 + yy + dy) * 9);
        rows |= r9 | (r9 >> 1);  // cell x holds point x or x + 1
      }
    word |= (rows & 0xFFu) << (8 * yy);
  }
  return word;
}

}  // namespace
}  // namespace yv
