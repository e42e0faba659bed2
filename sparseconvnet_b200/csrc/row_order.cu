// The order in which the output rows of a dense rulebook are packed into tensor-core tiles.
//
// A tile of 128 output rows costs one step per filter offset for which ANY of its rows has a rule, so rows
// that share the same set of offsets belong in the same tile.  In coordinate order a tile of an indoor scan
// (9 rules per row, 27 offsets) meets 22 to 25 offsets; with the rows sorted by their offset set ("mask") it
// meets 9.5 to 12.  The sort is stable, so rows of one mask stay in coordinate order and neighbouring rows of
// a tile still gather neighbouring input rows.  Only the packing changes: every output row is computed with
// its own rules, in the same offset order, and stored at its own place.
//
// Offsets of a tile of 128 rows, coordinate order -> sorted (counted on the synthetic workloads):
//   rooms, finest level (405 k rows) 22.4 -> 9.5      rooms, two levels down (37 k rows) 23.8 -> 10.3
//   shells and planes (267 k rows)   26.5 -> 13.8     4-D moving shells, 81 offsets      71.8 -> 35.2
//   stride-2 transposed layers (8 offsets, one rule per row): -> 1
//
// Steps: k_order_keys (mask -> sort key, and the digit counts of the first pass), then one stable counting pass per
// digit of at most nine bits (k_order_scatter, with k_order_count between two passes), then k_order_tiles: the union
// of the masks of every 128 rows, and the table's entries of those rows laid out one after the other.  Rows of one tile
// lie far apart in the table (52 to 99 sectors per 128 entries): looked up by the convolutions themselves, that was as
// much traffic as a quarter to a half of the rows they gather, once per layer.
#include <stdlib.h>

#include <algorithm>

#include "metadata.cuh"

namespace scn {
namespace {

constexpr int kTile = kOrderTile;
constexpr int kMaxDigit = 512;  // nine bits
constexpr int kThreads = 1024, kWarps = kThreads / 32;

template <typename KEY>
struct KeyBits {
  KEY bit[sizeof(KEY) == 4 ? 32 : kOrderMaxOffsets];  // what an offset with a rule sets in the sort key
};

// One more row with digit d in the block's counts: most rows of a surface share a handful of masks, so one update per
// distinct digit in the warp.
__device__ __forceinline__ void count_digit(int *h, int d) {
  const unsigned peers = __match_any_sync(__activemask(), d);
  if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&h[d], __popc(peers));
}
__device__ __forceinline__ void store_counts(const int *h, int R, int *block_count) {
  for (int i = threadIdx.x; i < R; i += kThreads) block_count[(long long)blockIdx.x * R + i] = h[i];
}

// Which offsets of a row have a rule (read from the table unless the rulebook's builder has left them in `known`), and
// the sort key made of them.
template <typename KEY, int WORDS>
__global__ void __launch_bounds__(kThreads)
k_order_keys(const int *__restrict__ nbr, const unsigned *__restrict__ known, long long n, int K, KeyBits<KEY> B,
             int rows_per_block, int R, KEY *__restrict__ keys, unsigned *__restrict__ masks,
             int *__restrict__ block_count, int *tiles_done) {
  SCN_GRID_WAIT();
  __shared__ int h[kMaxDigit];
  if (blockIdx.x == 0 && threadIdx.x == 0) *tiles_done = 0;  // (for k_order_tiles)
  for (int i = threadIdx.x; i < R; i += kThreads) h[i] = 0;
  __syncthreads();
  const long long r0 = (long long)blockIdx.x * rows_per_block, r1 = min(n, r0 + rows_per_block);
  for (long long r = r0 + threadIdx.x; r < r1; r += kThreads) {
    KEY key = 0;
#pragma unroll
    for (int w = 0; w < WORDS; ++w) {
      unsigned m = 0;
      if (known) {
        m = __ldg(known + r * WORDS + w);
      } else {
#pragma unroll 1
        for (int b0 = 0; b0 < 32 && w * 32 + b0 < K; b0 += 8) {
          int v[8];
#pragma unroll
          for (int b = 0; b < 8; ++b) v[b] = w * 32 + b0 + b < K ? __ldg(nbr + (long long)(w * 32 + b0 + b) * n + r) : -1;
#pragma unroll
          for (int b = 0; b < 8; ++b) m |= v[b] >= 0 ? 1u << (b0 + b) : 0u;
        }
        masks[r * WORDS + w] = m;
      }
#pragma unroll
      for (int b = 0; b < 32; ++b)
        if (m >> b & 1u) key |= B.bit[w * 32 + b];
    }
    keys[r] = key;
    count_digit(h, (int)key & (R - 1));
  }
  __syncthreads();
  store_counts(h, R, block_count);
}

// Digit counts of every block's rows (block_count [blocks][R]).
template <typename KEY>
__global__ void __launch_bounds__(kThreads)
k_order_count(const KEY *__restrict__ keys, long long n, int rows_per_block, int shift, int R,
              int *__restrict__ block_count) {
  SCN_GRID_WAIT();
  __shared__ int h[kMaxDigit];
  for (int i = threadIdx.x; i < R; i += kThreads) h[i] = 0;
  __syncthreads();
  const long long r0 = (long long)blockIdx.x * rows_per_block, r1 = min(n, r0 + rows_per_block);
  for (long long r = r0 + threadIdx.x; r < r1; r += kThreads) count_digit(h, (int)(keys[r] >> shift) & (R - 1));
  __syncthreads();
  store_counts(h, R, block_count);
}

// Stable scatter of a block's rows by one digit.  A block's first position of digit d is (rows of smaller
// digits) + (rows of digit d in the blocks before it), both added up from the blocks' counts (the last block reads as many
// of them as all do: totals of their own, cleared by a launch and added to by atomics, saved nothing); within the block the
// warps own consecutive segments.  rows_in null: the row of position i is i.
template <typename KEY>
__global__ void __launch_bounds__(kThreads)
k_order_scatter(const KEY *__restrict__ keys, const int *__restrict__ rows_in, long long n, int rows_per_block,
                int shift, int R, const int *__restrict__ block_count, KEY *__restrict__ keys_out, int *__restrict__ rows_out) {
  SCN_GRID_WAIT();
  __shared__ unsigned short cnt[kWarps][kMaxDigit];  // rows of digit d in warp w's segment, then in the warps before it
  __shared__ int base[kMaxDigit], part[kMaxDigit], part_total[kMaxDigit];  // (a block has fewer than 65536 rows)
  __shared__ int warp_sum[kWarps];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < kWarps * kMaxDigit / 2; i += kThreads) reinterpret_cast<unsigned *>(&cnt[0][0])[i] = 0;
  __syncthreads();
  const int seg = rows_per_block / kWarps;  // a multiple of 32
  const long long s0 = (long long)blockIdx.x * rows_per_block + (long long)warp * seg;
  const long long s1 = min(n, s0 + seg);
  // all 32 lanes together to the end (digit -1 past it): the counts are plain additions by one lane per digit, and the
  // places handed out below are in lane order
  for (long long c0 = s0; c0 < s1; c0 += 32) {
    const int d = c0 + lane < s1 ? (int)(keys[c0 + lane] >> shift) & (R - 1) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    if (d >= 0 && lane == __ffs(peers) - 1) cnt[warp][d] += (unsigned short)__popc(peers);
    __syncwarp();
  }
  // rows of digit d in the blocks before this one and in all: two threads per digit, every other block each
  const int d = tid & (kMaxDigit - 1), half = tid / kMaxDigit;
  int before = 0, tot = 0;
  if (d < R) {
#pragma unroll 16
    for (int b = half; b < (int)gridDim.x; b += 2) {
      const int c = __ldg(block_count + (long long)b * R + d);
      tot += c;
      before += b < (int)blockIdx.x ? c : 0;
    }
    if (half) part[d] = before, part_total[d] = tot;
  }
  __syncthreads();
  tot = half == 0 && d < R ? tot + part_total[d] : 0;
  int incl = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  if (half == 0 && d < R) {
    int at = incl - tot + before + part[d];
    for (int w = 0; w < warp; ++w) at += warp_sum[w];
    base[d] = at;
    unsigned run = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const unsigned c = cnt[w][d];
      cnt[w][d] = (unsigned short)run;
      run += c;
    }
  }
  __syncthreads();
  for (long long c0 = s0; c0 < s1; c0 += 32) {
    const long long r = c0 + lane;
    const bool here = r < s1;
    const KEY key = here ? keys[r] : 0;
    const int dg = here ? (int)(key >> shift) & (R - 1) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, dg);
    const int pos = here ? base[dg] + cnt[warp][dg] + __popc(peers & ((1u << lane) - 1u)) : 0;
    __syncwarp();
    if (here && lane == __ffs(peers) - 1) cnt[warp][dg] += (unsigned short)__popc(peers);
    __syncwarp();
    if (!here) continue;
    if (keys_out) keys_out[pos] = key;
    rows_out[pos] = rows_in ? rows_in[r] : (int)r;
  }
}

// Levels too small to sort: the identity order, its tiles and their entries in one launch, one block per tile.  Bound by trips to
// memory one behind the other: with at most 32 offsets a row's entries are asked for at once and stay in registers (2.8 us for
// 27 offsets on 6 k rows; 5.8 when they were read nine at a time, twice).
template <bool ONE_WORD>
__global__ void __launch_bounds__(kTile)
k_order_plain(const int *__restrict__ nbr, long long n, int K, int words, int *__restrict__ order,
              unsigned *__restrict__ tile_bits, int *__restrict__ packed) {
  SCN_GRID_WAIT();
  __shared__ unsigned bits[4];
  const long long t = blockIdx.x, p = t * kTile + threadIdx.x;
  if (ONE_WORD) {
    int v[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = k < K && p < n ? __ldg(nbr + (long long)k * n + p) : -1;
    if (threadIdx.x < 4) bits[threadIdx.x] = 0;
    order[p] = p < n ? (int)p : -1;
    __syncthreads();
    unsigned mine = 0;
#pragma unroll
    for (int k = 0; k < 32; ++k) mine |= v[k] >= 0 ? 1u << k : 0u;
    const unsigned seen = __reduce_or_sync(0xffffffffu, mine);
    if ((threadIdx.x & 31) == 0) atomicOr(&bits[0], seen);
    __syncthreads();
    const unsigned all = bits[0];
    if (threadIdx.x == 0) tile_bits[t] = all;
    int *dst = packed + t * K * kTile + threadIdx.x;
#pragma unroll
    for (int k = 0; k < 32; ++k)
      if (all >> k & 1u) dst[__popc(all & ((1u << k) - 1u)) * kTile] = v[k];
    return;
  }
  if (threadIdx.x < 4) bits[threadIdx.x] = 0;
  order[p] = p < n ? (int)p : -1;
  __syncthreads();
  unsigned seen = 0;  // of the current word, by this warp
#pragma unroll 9
  for (int k = 0; k < K; ++k) {
    const int v = p < n ? __ldg(nbr + (long long)k * n + p) : -1;
    if (__any_sync(0xffffffffu, v >= 0)) seen |= 1u << (k & 31);
    if ((k & 31) == 31 || k == K - 1) {
      if ((threadIdx.x & 31) == 0 && seen) atomicOr(&bits[k >> 5], seen);
      seen = 0;
    }
  }
  __syncthreads();
  int *dst = packed + t * K * kTile + threadIdx.x;
  for (int w = 0; w < words; ++w) {
    const unsigned all = bits[w];
    if (threadIdx.x == 0) tile_bits[t * words + w] = all;
#pragma unroll 4
    for (unsigned u = all; u; u &= u - 1) {
      const int k = w * 32 + __ffs(u) - 1;
      *dst = p < n ? __ldg(nbr + (long long)k * n + p) : -1;
      dst += kTile;
    }
  }
}

// Fine rows with one rule each (a Deconvolution whose filter is its stride) by the offset of that rule, from the table as the
// Convolution has it (nbr [K][n_out] = fine row or -1) and the rules per offset that its builder has counted: whole tiles
// of one offset, -1 behind an offset's last row.  A block takes a run of the offset's places for its coarse rows, so the
// blocks come in the order in which they get there; what a row's sum is does not depend on the tile it is in.  The block
// that finishes last clears the cursors, so that the launch can be repeated (a graph that has recorded it).  One launch
// where the transposed table, its masks, a counting pass and the tiles were six: 17 us per level on small levels, 95 on
// 1.6 M rows, now 5 and 14.
__global__ void __launch_bounds__(256)
k_order_children(const int *__restrict__ nbr, long long n_out, int K, const unsigned long long *__restrict__ counts,
                 unsigned long long *cursors, long long n_tiles, int *__restrict__ order, unsigned *__restrict__ tile_bits,
                 int *__restrict__ packed) {
  SCN_GRID_WAIT();
  __shared__ int start[kChildrenMaxOffsets + 1];  // first tile of an offset
  __shared__ int before[8][kChildrenMaxOffsets];  // rules of an offset in this warp's coarse rows, then in the warps before
  __shared__ long long base[kChildrenMaxOffsets];
  static_assert(kChildrenMaxOffsets == 32, "a lane per offset");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    const int tiles = lane < K ? (int)((counts[lane] + kTile - 1) / kTile) : 0;
    int incl = tiles;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += u;
    }
    start[lane] = incl - tiles;
    if (lane == 31) start[32] = incl;
  }
  const long long o = (long long)blockIdx.x * 256 + tid;
#pragma unroll 8
  for (int k = 0; k < K; ++k) {
    const unsigned hits = __ballot_sync(0xffffffffu, o < n_out && __ldg(nbr + k * n_out + o) >= 0);
    if (lane == 0) before[warp][k] = __popc(hits);
  }
  __syncthreads();
  if (tid < K) {
    int run = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const int c = before[w][tid];
      before[w][tid] = run;
      run += c;
    }
    base[tid] = run ? (long long)atomicAdd(&cursors[tid], (unsigned long long)run) : 0;
  }
  __syncthreads();
#pragma unroll 8
  for (int k = 0; k < K; ++k) {
    const int v = o < n_out ? __ldg(nbr + k * n_out + o) : -1;
    const unsigned hits = __ballot_sync(0xffffffffu, v >= 0);
    const long long at = base[k] + before[warp][k] + __popc(hits & ((1u << lane) - 1u));
    if (v >= 0 && at < (long long)counts[k]) {
      const long long p = (long long)start[k] * kTile + at;
      order[p] = v;
      packed[p / kTile * K * kTile + p % kTile] = (int)o;
    }
  }
  for (long long t = o; t < n_tiles; t += (long long)gridDim.x * 256) {
    unsigned bits = 0;
    for (int k = 0; k < K; ++k)
      if (t >= start[k] && t < start[k + 1]) bits = 1u << k;
    tile_bits[t] = bits;
  }
  if (blockIdx.x == 0)
    for (int k = warp; k <= K; k += 8) {  // behind the last row of an offset, and of all
      const long long p0 = k < K ? (long long)start[k] * kTile + (long long)counts[k] : (long long)start[K] * kTile;
      const long long p1 = k < K ? (long long)start[k + 1] * kTile : n_tiles * kTile;
      for (long long p = p0 + lane; p < p1; p += 32) {
        order[p] = -1;
        packed[p / kTile * K * kTile + p % kTile] = -1;
      }
    }
  __syncthreads();
  if (tid == 0 && atomicAdd(&cursors[K], 1ull) == (unsigned long long)gridDim.x - 1)
    for (int k = 0; k <= K; ++k) cursors[k] = 0;
}

// The tiles by how many offsets they have, most first, stable (run by one block of 256 threads, the last of k_order_tiles to
// pack its own: it adds 4 us to 21 us at 300 k rows).  Handed out in ascending order of their masks the tiles left the
// busiest SM 1.1 to 1.7 times the average; most offsets first, back and forth over the CTAs, 1.02 to 1.2: 32 -> 32 planes
// on 1.6 M rows 335 -> 317 us, 96 -> 96 on 155 k rows 169 -> 133 us.  Below 149 tiles no CTA has two; from 65536 on the
// counts would not fit their 16 bits and each CTA has hundreds of tiles, which is balance enough.
constexpr int kWorkBins = 32;
template <int WORDS>
__device__ void tiles_by_work(const unsigned *tile_bits, int n_tiles, int K, int *by_work) {
  __shared__ __align__(16) unsigned short hist[kWorkBins][256];
  __shared__ int bin_sum[kWorkBins];
  static_assert(kWorkBins == 32, "a lane per bin");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (n_tiles + 255) / 256, t0 = min(n_tiles, tid * per), t1 = min(n_tiles, t0 + per);
  const unsigned scale = ((unsigned)kWorkBins << 16) / (unsigned)(K + 1);
  // each tile of the thread's run in order, sixteen masks on their way (the block works alone: every trip to L2 shows);
  // the bins of a run of up to sixteen stay in registers for the second walk
  int b[16];
  auto load = [&](int t) {
    unsigned bits[16][WORDS];
#pragma unroll
    for (int i = 0; i < 16; ++i)
#pragma unroll
      for (int w = 0; w < WORDS; ++w) bits[i][w] = t + i < t1 ? __ldcg(tile_bits + (long long)(t + i) * WORDS + w) : 0u;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      unsigned c = 0;
#pragma unroll
      for (int w = 0; w < WORDS; ++w) c += __popc(bits[i][w]);
      b[i] = (kWorkBins - 1) - (int)(c * scale >> 16);
    }
  };
  auto each = [&](bool again, auto use) {
    for (int t = t0; t < t1; t += 16) {
      if (!again || per > 16) load(t);
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (t + i < t1) use(t + i, b[i]);
    }
  };
#pragma unroll
  for (int b = 0; b < kWorkBins; ++b) hist[b][tid] = 0;
  each(false, [&](int, int b) { ++hist[b][tid]; });
  __syncthreads();
  // exclusive sums over (bin, thread): a warp has four bins, a lane eight neighbouring threads' counts of each
  int before[4];
  uint4 v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[i] = *reinterpret_cast<const uint4 *>(&hist[warp * 4 + i][lane * 8]);
    const unsigned pairs = v[i].x + v[i].y + v[i].z + v[i].w;  // (no half overflows: fewer than 65536 tiles)
    const int sum = (int)(pairs & 0xFFFFu) + (int)(pairs >> 16);
    int incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += u;
    }
    before[i] = incl - sum;
    if (lane == 31) bin_sum[warp * 4 + i] = incl;
  }
  __syncthreads();
  int base = bin_sum[lane], own = base;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, base, d);
    if (lane >= d) base += u;
  }
  base -= own;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    unsigned at = (unsigned)(before[i] + __shfl_sync(0xffffffffu, base, warp * 4 + i));
    unsigned *w = reinterpret_cast<unsigned *>(&v[i]);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const unsigned lo = w[e] & 0xFFFFu, hi = w[e] >> 16;
      w[e] = (at & 0xFFFFu) | ((at + lo) << 16);
      at += lo + hi;
    }
    *reinterpret_cast<uint4 *>(&hist[warp * 4 + i][lane * 8]) = v[i];
  }
  __syncthreads();
  each(true, [&](int t, int b) { by_work[hist[b][tid]++] = t; });
}

// Two tiles per block, a row per thread: tile_bits, packed, and -1 in the order array past the last row.  Bound by the trips to
// L2 that the entries of rows far apart take, so many threads with eight of them on their way.  (A warp per tile, four rows
// per lane: 104 us for the eleven sorted levels of one room where this takes 67, 25.7 and 22.3 on 267 k rows, 377 and 347 on
// 1.5 M rows with 81 offsets.)
template <int WORDS>
__global__ void __launch_bounds__(256)
k_order_tiles(int *__restrict__ order, long long n, int K, const int *__restrict__ nbr, const unsigned *__restrict__ masks,
              unsigned *tile_bits, int *__restrict__ packed, long long n_tiles, int *by_work, int *done) {
  SCN_GRID_WAIT();
  __shared__ unsigned warp_bits[8][WORDS];
  static_assert(kTile == 128, "a row per thread, four warps per tile");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, in_tile = threadIdx.x & (kTile - 1);
  const long long t = (long long)blockIdx.x * 2 + threadIdx.x / kTile;
  int row = -1;
  unsigned m[WORDS];
  if (t < n_tiles) {
    const long long p = t * kTile + in_tile;
    if (p < n) row = order[p];
    else order[p] = -1;
  }
#pragma unroll
  for (int w = 0; w < WORDS; ++w) m[w] = row >= 0 ? __ldg(masks + (long long)row * WORDS + w) : 0u;
#pragma unroll
  for (int w = 0; w < WORDS; ++w) {
    const unsigned any = __reduce_or_sync(0xffffffffu, m[w]);
    if (lane == 0) warp_bits[warp][w] = any;
  }
  __syncthreads();
  if (t < n_tiles) {
    int *dst = packed + t * K * kTile + in_tile;
    const int w0 = warp & ~3;
#pragma unroll
    for (int w = 0; w < WORDS; ++w) {
      const unsigned all = warp_bits[w0][w] | warp_bits[w0 + 1][w] | warp_bits[w0 + 2][w] | warp_bits[w0 + 3][w];
      if (in_tile == 0) tile_bits[t * WORDS + w] = all;
      unsigned u = all;
      while (u) {  // eight offsets at a time
        int v[8];
        unsigned left = u;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int b = left ? __ffs(left) - 1 : 0;
          v[e] = left && (m[w] >> b & 1u) ? __ldg(nbr + (long long)(w * 32 + b) * n + row) : -1;
          left &= left - 1;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (u) {
            *dst = v[e];
            dst += kTile;
            u &= u - 1;
          }
      }
    }
  }
  if (!by_work) return;
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(done, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (last) tiles_by_work<WORDS>(tile_bits, (int)n_tiles, K, by_work);
}

// Which key bits the offsets set, and how many bits there are.  Fewer bits cost fewer passes,
// and below about 65 000 rows a coarser key also packs better, because full masks are hardly ever repeated.  Offsets
// per tile of 128 rows on rooms of 405 k / 119 k / 37 k / 15 k rows, 27 offsets (in coordinate order 22.4 / 23.9 /
// 23.8 / 25.6):
//   27 bits, the first offset highest               9.48   9.88  10.3  17.3   three passes
//   the 12 edges, then the 6 faces                   9.70  10.2   11.4  18.1   two
//   OR-ed over the middle dimension (9 bits)        13.0   12.8   11.3  14.4   one
// A 4-D filter of size 3 (81 offsets, nearly every site of moving shells has a mask of its own): for the earlier and the
// later time slice whether any offset with x (y, z) = -1, 0, 1 has a rule, then the slice of the site itself OR-ed over
// y: 27 bits, 36.7 offsets per tile; all 81 bits in filter order 40.8; the time slices OR-ed over y and the middle one in
// full 35.2, but the rows of a tile lie a third farther apart.  Other large filters: groups of consecutive offsets.
// An offset may set several bits: bit[k] is their union.
int key_bits(const Rulebook &rb, int K, long long n, unsigned long long *bit) {
  for (int k = 0; k < K; ++k) bit[k] = 0;
  bool three = rb.dim >= 3;
  for (int d = 0; d < rb.dim; ++d) three &= rb.filter[d] == 3;
  if (rb.dim == 3 && three && n < 65536) {
    for (int k = 0; k < 27; ++k) bit[k] = 1ull << (8 - ((k / 9) * 3 + k % 3));
    return 9;
  }
  if (rb.dim == 3 && three && n < 524288) {
    int edges = 0, faces = 0;
    for (int k = 0; k < 27; ++k) {
      const int far = (k % 3 != 1) + (k / 3 % 3 != 1) + (k / 9 != 1);
      if (far == 2) bit[k] = 1ull << (17 - edges++);
      if (far == 1) bit[k] = 1ull << (5 - faces++);
    }
    return 18;
  }
  if (K <= 32) {
    for (int k = 0; k < K; ++k) bit[k] = 1ull << (K - 1 - k);
    return K;
  }
  if (rb.dim == 4 && three) {
    for (int k = 0; k < 81; ++k) {
      const int t = k % 3, z = (k / 3) % 3, y = (k / 9) % 3, x = k / 27;
      if (t == 1)
        bit[k] = 1ull << (8 - (x * 3 + z));
      else
        bit[k] = ((1ull << (8 - x)) | (1ull << (5 - y)) | (1ull << (2 - z))) << (t == 0 ? 18 : 9);
    }
    return 27;
  }
  const int most = n >= 262144 ? 45 : 27, group = (K + most - 1) / most, bits = (K + group - 1) / group;
  for (int k = 0; k < K; ++k) bit[k] = 1ull << (bits - 1 - k / group);
  return bits;
}

template <typename KEY, int WORDS>
int build(const int *table, const unsigned *known, long long n, int K, const unsigned long long *bit, int bits, RowOrder &ord, cudaStream_t stream) {
  Scratch tmp(stream);
  unsigned *masks = nullptr;
  KEY *keys[2] = {nullptr, nullptr};
  int *rows = nullptr, *counts = nullptr;
  const int passes = (bits + 8) / 9, digit = (bits + passes - 1) / passes, R = 1 << digit;
  // Rows per block: a multiple of the warps' 32-row chunks; one block per SM at most, because a block adds up the counts
  // of the blocks before it itself
  const long long rpb = std::min<long long>(ceil_div(ceil_div(n, 148), kThreads), 63) * kThreads;
  const int blocks = (int)ceil_div(n, rpb);
  KeyBits<KEY> B{};
  for (int k = 0; k < K; ++k) B.bit[k] = (KEY)bit[k];
  if (!known) SCN_TRY(tmp.get(&masks, sizeof(unsigned) * WORDS * (size_t)n));
  SCN_TRY(tmp.get(&keys[0], sizeof(KEY) * (size_t)n));
  SCN_TRY(tmp.get(&counts, sizeof(int) * ((size_t)blocks * R + 1)));  // and the blocks that have packed their tiles
  int *const done = counts + (size_t)blocks * R;
  if (passes > 1) {
    SCN_TRY(tmp.get(&keys[1], sizeof(KEY) * (size_t)n));
    SCN_TRY(tmp.get(&rows, sizeof(int) * (size_t)n));
  }
  if (ord.n_tiles > 148 && ord.n_tiles < 65536) SCN_TRY(device_alloc((void **)&ord.by_work, sizeof(int) * (size_t)ord.n_tiles, stream));
  SCN_LAUNCH((k_order_keys<KEY, WORDS>), blocks, kThreads, 0, stream, table, known, n, K, B, (int)rpb, R, keys[0], masks, counts, done);
  const int *src = nullptr;
  for (int p = 0; p < passes; ++p) {
    int *dst = ((passes - 1 - p) & 1) ? rows : ord.order;  // alternating so that the last pass writes ord.order
    KEY *kin = keys[p & 1], *kout = p + 1 < passes ? keys[(p + 1) & 1] : nullptr;
    if (p > 0)
      SCN_LAUNCH((k_order_count<KEY>), blocks, kThreads, 0, stream, kin, n, (int)rpb, p * digit, R, counts);
    SCN_LAUNCH((k_order_scatter<KEY>), blocks, kThreads, 0, stream, kin, src, n, (int)rpb, p * digit, R, counts, kout, dst);
    src = dst;
  }
  SCN_LAUNCH((k_order_tiles<WORDS>), (unsigned)ceil_div(ord.n_tiles, 2), 256, 0, stream, ord.order, n, K, table, known ? known : masks, ord.tile_bits, ord.packed, ord.n_tiles, ord.by_work, done);
  SCN_CUDA_CHECK(cudaGetLastError());
  return SCN_OK;
}

}  // namespace

void free_row_order(RowOrder &o, cudaStream_t stream) {
  device_free(o.order, stream);
  device_free(o.tile_bits, stream);
  device_free(o.packed, stream);
  device_free(o.by_work, stream);
  o = RowOrder{};
}

int rulebook_children_order(const Rulebook &rb, RowOrder &ord, cudaStream_t stream) {
  if (ord.order || rb.n_in == 0) return SCN_OK;
  const int K = rb.n_offsets;
  SCN_REQUIRE(rb.one_parent && K <= kChildrenMaxOffsets && rb.n_in < (1ll << 31), SCN_ERR_UNSUPPORTED, "children order: %d offsets", K);
  RowOrder o;
  o.words = 1;
  o.one_offset = true;
  o.n_tiles = (rb.n_in + (long long)K * (kTile - 1)) / kTile;  // every offset's last tile may be nearly empty
  int st = device_alloc((void **)&o.order, sizeof(int) * (size_t)o.n_tiles * kTile, stream);
  if (st == SCN_OK) st = device_alloc((void **)&o.tile_bits, sizeof(unsigned) * (size_t)o.n_tiles, stream);
  if (st == SCN_OK) st = device_alloc((void **)&o.packed, sizeof(int) * (size_t)o.n_tiles * K * kTile, stream);
  if (st == SCN_OK) {
    SCN_LAUNCH(k_order_children, (unsigned)std::max<long long>(1, ceil_div(rb.n_out, 256)), 256, 0, stream, rb.nbr, rb.n_out, K, rb.counts_dev, rb.counts_dev + K + 1, o.n_tiles, o.order, o.tile_bits, o.packed);
    if (cudaGetLastError() != cudaSuccess) {
      set_error("children order: launch failed");
      st = SCN_ERR_CUDA;
    }
  }
  if (st != SCN_OK) {
    free_row_order(o, stream);
    return st;
  }
  ord = o;
  return SCN_OK;
}

// Builds the packing order of a rulebook table [K][n] if it is not there yet.
int rulebook_row_order(const Rulebook &rb, const int *table, long long n, RowOrder &ord, cudaStream_t stream) {
  if (ord.order || n == 0) return SCN_OK;
  const int K = rb.n_offsets;
  SCN_REQUIRE(K >= 1 && K <= kOrderMaxOffsets && n < (1ll << 31), SCN_ERR_UNSUPPORTED, "row order: %d offsets", K);
  RowOrder o;
  o.words = K <= 32 ? 1 : 4;
  o.n_tiles = ceil_div(n, kTile);
  int st = device_alloc((void **)&o.order, sizeof(int) * (size_t)o.n_tiles * kTile, stream);
  if (st == SCN_OK) st = device_alloc((void **)&o.tile_bits, sizeof(unsigned) * (size_t)o.words * o.n_tiles, stream);
  if (st == SCN_OK) st = device_alloc((void **)&o.packed, sizeof(int) * (size_t)o.n_tiles * K * kTile, stream);
  // Small levels are bound by latency whatever the order, and the sort takes as long as one of their layers.
  long long least = 8192;
  if (const char *e = getenv("SCN_ORDER_MIN_ROWS")) least = atoll(e);
  if (st == SCN_OK && n < least) {
    SCN_LAUNCH((K <= 32 ? k_order_plain<true> : k_order_plain<false>), (unsigned)o.n_tiles, kTile, 0, stream, table, n, K, o.words, o.order, o.tile_bits, o.packed);
    if (cudaGetLastError() != cudaSuccess) {
      set_error("row order: launch failed");
      st = SCN_ERR_CUDA;
    }
  } else if (st == SCN_OK) {
    unsigned long long bit[kOrderMaxOffsets];
    const int bits = key_bits(rb, K, n, bit);
    const unsigned *known = table == rb.nbr ? rb.masks : nullptr;
    st = K <= 32 ? build<unsigned, 1>(table, known, n, K, bit, bits, o, stream)
                 : build<unsigned long long, 4>(table, known, n, K, bit, bits, o, stream);
  }
  if (st != SCN_OK) {
    free_row_order(o, stream);
    return st;
  }
  ord = o;
  return SCN_OK;
}

}  // namespace scn
