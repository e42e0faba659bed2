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

constexpr int kStepWarps = 4;  // producing warps of a step: 32 rows each
constexpr int kRecords = 4;    // items the entries run ahead of the roles that store results

// What the roles behind the entries have to know of an item: its steps, its tile (the last one too, so that the rows of the
// item behind it can be asked for early), which part of the tile's offsets or which column block it is.
struct ItemRecord {
  int steps, tile, part, next_tile;
};

// The tile of an item: the tiles with the most offsets first (packed tiles come in ascending order of their masks, so from
// the back where they have not been sorted by work).  Past the last item any tile.
template <class Params>
__device__ __forceinline__ int item_tile(const Params &P, long long item) {
  if (item >= P.n_items) return 0;
  const int i = P.per_tile == 1 ? (int)item : (int)item / P.per_tile;
  return P.by_work ? __ldg(P.by_work + i) : (int)P.n_tiles - 1 - i;
}

// The tiles of a CTA's items in turn: the tile of an item is asked for three items ahead and its mask of offsets one ahead, so
// that neither trip to memory is waited for between two tiles.
template <class Params>
struct Tiles {
  int tile, next, next2;
  unsigned mask[4], next_mask[4];
  __device__ __forceinline__ void fetch(const Params &P, int t, unsigned (&m)[4]) {
#pragma unroll
    for (int w = 0; w < 4; ++w) m[w] = w < P.words ? __ldg(P.tile_bits + (long long)t * P.words + w) : 0u;
  }
  __device__ __forceinline__ void start(const Params &P) {
    tile = item_tile(P, item_of(0)), next = item_tile(P, item_of(1)), next2 = item_tile(P, item_of(2));
    fetch(P, tile, mask);
    fetch(P, next, next_mask);
  }
  // from item `it` to the one behind it
  __device__ __forceinline__ void advance(const Params &P, long long it) {
    tile = next, next = next2, next2 = item_tile(P, item_of(it + 3));
#pragma unroll
    for (int w = 0; w < 4; ++w) mask[w] = next_mask[w];
    fetch(P, next, next_mask);
  }
};

// What the bulk copies of a CTA have been ordered for, left by the threads that order them when they leave their loops.
struct OrderedCopies {
  int slots;     // by the entries, the slots that end the work among them
  int slabs[2];  // weights of the steps g, g + groups, ... by group g of the producing warps
};

// The last step of those that use stage `st` whose slab has been ordered, -1: none.  (The ones before it have been consumed: an order
// waits for that.)
__host__ __device__ inline int last_slab(const int *slabs, int groups, int n_stages, int st) {
  int last = -1;
  for (int g = 0; g < groups; ++g)
    for (int i = slabs[g] - 1; i >= 0 && i >= slabs[g] - n_stages; --i)
      if ((g + i * groups) % n_stages == st) {
        if (g + i * groups > last) last = g + i * groups;
        break;
      }
  return last;
}

// A CTA whose roles left early, whichever of them and on whichever way: its bulk copies must land before its shared memory goes
// away.  All threads come here behind the block's last barrier, when nobody orders any more; one waits for each slot and each stage.
template <int SLOTS>
__device__ __forceinline__ void land_slots(unsigned long long (&s_full)[SLOTS], int slots) {
  const int si = threadIdx.x, uses = (slots + SLOTS - 1 - si) / SLOTS;
  if (si < SLOTS && uses > 0) mbar_wait(&s_full[si], (unsigned)((uses - 1) & 1));
}
template <class Control>
__device__ __forceinline__ void land_copies(Control &C, int n_stages, int groups) {
  land_slots(C.s_full, C.ordered.slots);
  const int st = (int)threadIdx.x - 32;
  if (st < 0 || st >= n_stages) return;
  const int step = last_slab(C.ordered.slabs, groups, n_stages, st);
  if (step >= 0) mbar_wait(&C.full[st], (unsigned)(step / n_stages & 1));
}
}  // namespace scn
