// What the tcgen05 kernels on mask-sorted row tiles share (conv_tile.cu, conv_six.cu): descriptors of the gathered rows, the
// instruction descriptor, the order in which a CTA takes its items.
#pragma once

#include "metadata.cuh"
#include "tc_ptx.cuh"

namespace scn {

int sum_partial_tiles(const float *partial, int n_split, long long n_pos, int cout, const int *order, long long n_out,
                      const float *bias, const float *bn_scale, const float *bn_shift, float leak, float *out,
                      cudaStream_t stream, unsigned char *out_split = nullptr, int out_sp = 1, int parts = 1);

// Operand descriptor of a stage of gathered rows: K-major, 128-, 64- or 32-byte swizzle (a row's 16-byte chunk c is
// stored at chunk c ^ (r & 7), c ^ ((r >> 1) & 3) or c ^ ((r >> 2) & 1)), 8-row groups back to back.  `offset`: bytes along the row.
// Whole rows being contiguous is what makes the gather fast: a row arrives as full 128-byte writes.  With the pieces
// spread over core matrices 2 KB apart every 16 bytes were a write of their own: 1 700 cycles per 16 KB step.
template <unsigned ROW>
__device__ __forceinline__ unsigned long long rows_desc(unsigned addr, unsigned offset) {
  unsigned long long d = 0;
  d |= (unsigned long long)(((addr + offset) >> 4) & 0x3FFF);
  d |= 1ull << 16;
  d |= (unsigned long long)((ROW * 8) >> 4) << 32;
  d |= 1ull << 46;
  d |= (unsigned long long)(ROW == 128 ? 2 : ROW == 64 ? 4 : 6) << 61;
  return d;
}

constexpr int kNoRules = 1 << 20;  // a slot of a tile without any rule: rows and weights of zeros

__host__ __device__ inline unsigned tile_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(kOrderTile >> 4) << 24);
}

// bits `lo` .. `hi` - 1 of the set bits of a 128-bit mask, counted from bit 0 (the offsets of one part of a split)
__device__ __forceinline__ void keep_range(unsigned (&m)[4], int lo, int hi) {
  int seen = 0;
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    unsigned keep = 0;
    for (unsigned u = m[w]; u; u &= u - 1, ++seen)
      if (seen >= lo && seen < hi) keep |= u & (0u - u);
    m[w] = keep;
  }
}

// The items of a CTA: back and forth over the CTAs, so that of items in descending order of work each gets about the same.
__device__ __forceinline__ long long item_of(long long it) {
  return it & 1 ? (it + 1) * gridDim.x - 1 - blockIdx.x : it * gridDim.x + blockIdx.x;
}
__device__ __forceinline__ long long items_here(long long n_items) {
  const long long full = n_items / gridDim.x;
  return full + (item_of(full) < n_items ? 1 : 0);
}
}  // namespace scn
