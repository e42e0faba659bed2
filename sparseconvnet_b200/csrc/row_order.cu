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
// Steps: k_order_keys (mask -> sort key of up to 64 bits), then one stable counting pass per digit of at most
// nine bits (k_order_count, k_order_scatter), then k_order_tiles (the union of the masks of every 128 rows).
#include <stdlib.h>

#include <algorithm>

#include "metadata.cuh"

namespace scn {
namespace {

constexpr int kTile = kOrderTile;
constexpr int kMaxDigit = 512;  // nine bits
constexpr int kCountThreads = 512, kScatterThreads = 512;

struct KeyBits {
  unsigned char pos[kOrderMaxOffsets];  // bit of the sort key that offset k sets; 255: none
};

// One thread per output row: which offsets have a rule, and the sort key made of them.
template <typename KEY, int WORDS>
__global__ void __launch_bounds__(256)
k_order_keys(const int *__restrict__ nbr, long long n, int K, KeyBits B, KEY *__restrict__ keys,
             unsigned *__restrict__ masks) {
  const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  KEY key = 0;
  unsigned m[WORDS];
#pragma unroll
  for (int w = 0; w < WORDS; ++w) m[w] = 0;
#pragma unroll
  for (int w = 0; w < WORDS; ++w) {
    if (w * 32 >= K) break;
#pragma unroll 8
    for (int b = 0; b < 32; ++b) {
      const int k = w * 32 + b;
      if (k < K && __ldg(nbr + (long long)k * n + r) >= 0) {
        m[w] |= 1u << b;
        if (B.pos[k] != 255) key |= (KEY)1 << B.pos[k];
      }
    }
  }
  keys[r] = key;
#pragma unroll
  for (int w = 0; w < WORDS; ++w) masks[r * WORDS + w] = m[w];
}

// Digit counts of every block's rows (block_count [blocks][R]) and of all rows (total [R], zeroed before).
template <typename KEY>
__global__ void __launch_bounds__(kCountThreads)
k_order_count(const KEY *__restrict__ keys, long long n, int rows_per_block, int shift, int R,
              int *__restrict__ block_count, int *__restrict__ total) {
  __shared__ int h[kMaxDigit];
  for (int i = threadIdx.x; i < R; i += blockDim.x) h[i] = 0;
  __syncthreads();
  const long long r0 = (long long)blockIdx.x * rows_per_block, r1 = min(n, r0 + rows_per_block);
  for (long long r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
    const int d = (int)(keys[r] >> shift) & (R - 1);
    // most rows of a surface share a handful of masks: one update per distinct digit in the warp
    const unsigned peers = __match_any_sync(__activemask(), d);
    if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&h[d], __popc(peers));
  }
  __syncthreads();
  for (int i = threadIdx.x; i < R; i += blockDim.x) {
    block_count[(long long)blockIdx.x * R + i] = h[i];
    if (h[i]) atomicAdd(&total[i], h[i]);
  }
}

// Stable scatter of a block's rows by one digit.  A block's first position of digit d is (rows of smaller
// digits) + (rows of digit d in the blocks before it), both read from the counts; within the block the warps
// own consecutive segments.  rows_in null: the row of position i is i.
template <typename KEY>
__global__ void __launch_bounds__(kScatterThreads)
k_order_scatter(const KEY *__restrict__ keys, const int *__restrict__ rows_in, long long n, int rows_per_block,
                int shift, int R, const int *__restrict__ block_count, const int *__restrict__ total,
                KEY *__restrict__ keys_out, int *__restrict__ rows_out) {
  constexpr int kWarps = kScatterThreads / 32;
  __shared__ int cnt[kWarps][kMaxDigit];  // then: next position of digit d for warp w
  __shared__ int warp_sum[kWarps];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < kWarps * kMaxDigit; i += kScatterThreads) (&cnt[0][0])[i] = 0;
  __syncthreads();
  const int seg = rows_per_block / kWarps;  // a multiple of 32
  const long long s0 = (long long)blockIdx.x * rows_per_block + (long long)warp * seg;
  const long long s1 = min(n, s0 + seg);
  for (long long r = s0 + lane; r < s1; r += 32) {
    const int d = (int)(keys[r] >> shift) & (R - 1);
    const unsigned peers = __match_any_sync(__activemask(), d);
    if (lane == __ffs(peers) - 1) cnt[warp][d] += __popc(peers);
    __syncwarp(__activemask());
  }
  // thread d: rows of digit d in the blocks before this one, and the exclusive scan of the totals
  int before = 0, tot = 0;
  if (tid < R) {
    tot = total[tid];
#pragma unroll 8
    for (int b = 0; b < (int)blockIdx.x; ++b) before += block_count[(long long)b * R + tid];
  }
  int incl = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  int base = incl - tot + before;
  for (int w = 0; w < warp; ++w) base += warp_sum[w];
  if (tid < R) {
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const int c = cnt[w][tid];
      cnt[w][tid] = base;
      base += c;
    }
  }
  __syncthreads();
  for (long long r = s0 + lane; r < s1; r += 32) {
    const unsigned act = __activemask();
    const KEY key = keys[r];
    const int d = (int)(key >> shift) & (R - 1);
    const unsigned peers = __match_any_sync(act, d);
    const int pos = cnt[warp][d] + __popc(peers & ((1u << lane) - 1u));
    __syncwarp(act);
    if (lane == __ffs(peers) - 1) cnt[warp][d] += __popc(peers);
    __syncwarp(act);
    if (keys_out) keys_out[pos] = key;
    rows_out[pos] = rows_in ? rows_in[r] : (int)r;
  }
}

// tile_bits[t][WORDS]: offsets for which any of the tile's rows has a rule; one warp per tile.  The order array
// is filled with -1 up to its padded length.
template <int WORDS>
__global__ void __launch_bounds__(256)
k_order_tiles(int *__restrict__ order, long long n, long long n_padded, const unsigned *__restrict__ masks,
              unsigned *__restrict__ tile_bits, long long n_tiles) {
  const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= n_tiles) return;
  unsigned m[WORDS];
#pragma unroll
  for (int w = 0; w < WORDS; ++w) m[w] = 0;
#pragma unroll
  for (int i = 0; i < kTile / 32; ++i) {
    const long long p = t * kTile + i * 32 + lane;
    if (p < n) {
      const long long r = order[p];
#pragma unroll
      for (int w = 0; w < WORDS; ++w) m[w] |= __ldg(masks + r * WORDS + w);
    } else if (p < n_padded) {
      order[p] = -1;
    }
  }
#pragma unroll
  for (int w = 0; w < WORDS; ++w) {
    const unsigned u = __reduce_or_sync(0xffffffffu, m[w]);
    if (lane == 0) tile_bits[t * WORDS + w] = u;
  }
}

__global__ void k_order_identity(int *order, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) order[i] = (int)i;
}

// Which key bit an offset sets.  Up to 32 offsets: one bit each, the first offset the highest (ordering by the
// leading offsets first keeps masks that differ in the trailing ones together: 9.5 offsets per tile of 128 rows
// on rooms; by how close an offset's frequency is to one half: 9.7).  More offsets: a 4-D filter of size 3 puts
// the offsets of the earlier and later time slice first, OR-ed over one spatial dimension, then the slice of the
// site itself in full (45 bits: 35.2 offsets per tile; all 81 bits in filter order: 40.8).  Other large filters:
// OR-ed over groups of consecutive offsets.
int key_bits(int dim, const int64_t *filter, int K, KeyBits &B) {
  for (int k = 0; k < kOrderMaxOffsets; ++k) B.pos[k] = 255;
  if (K <= 32) {
    for (int k = 0; k < K; ++k) B.pos[k] = (unsigned char)(K - 1 - k);
    return K;
  }
  if (dim == 4 && filter && filter[0] == 3 && filter[1] == 3 && filter[2] == 3 && filter[3] == 3) {
    for (int k = 0; k < 81; ++k) {
      const int t = k % 3, z = (k / 3) % 3, y = (k / 9) % 3, x = k / 27;
      int rank;  // 0 = highest bit
      if (t == 1)
        rank = 18 + (x * 3 + y) * 3 + z;
      else
        rank = (t == 0 ? 0 : 9) + x * 3 + z;
      B.pos[k] = (unsigned char)(44 - rank);
    }
    return 45;
  }
  const int group = (K + 44) / 45, bits = (K + group - 1) / group;
  for (int k = 0; k < K; ++k) B.pos[k] = (unsigned char)(bits - 1 - k / group);
  return bits;
}

struct Scratch {  // freed on every way out
  void *p[8] = {nullptr};
  int n = 0;
  cudaStream_t stream;
  explicit Scratch(cudaStream_t s) : stream(s) {}
  ~Scratch() {
    for (int i = 0; i < n; ++i) device_free(p[i], stream);
  }
  int get(void **q, size_t bytes) {
    SCN_TRY(device_alloc(q, bytes, stream));
    p[n++] = *q;
    return SCN_OK;
  }
};

template <typename KEY, int WORDS>
int build(const int *table, long long n, int K, const KeyBits &B, int bits, RowOrder &ord, bool sort, cudaStream_t stream) {
  Scratch tmp(stream);
  unsigned *masks = nullptr;
  KEY *keys[2] = {nullptr, nullptr};
  int *rows = nullptr, *counts = nullptr, *totals = nullptr;
  SCN_TRY(tmp.get((void **)&masks, sizeof(unsigned) * WORDS * (size_t)n));
  SCN_TRY(tmp.get((void **)&keys[0], sizeof(KEY) * (size_t)n));
  SCN_LAUNCH((k_order_keys<KEY, WORDS>), (unsigned)ceil_div(n, 256), 256, 0, stream, table, n, K, B, keys[0], masks);
  if (!sort) {
    SCN_LAUNCH(k_order_identity, (unsigned)ceil_div(n, 256), 256, 0, stream, ord.order, n);
  } else {
    const int passes = (bits + 8) / 9, digit = (bits + passes - 1) / passes, R = 1 << digit;
    // Rows per block: a multiple of the warps' 32-row chunks; at most about 200 blocks, because a block adds up the
    // counts of the blocks before it itself
    long long rpb = ceil_div(ceil_div(n, 200), kScatterThreads) * kScatterThreads;
    const int blocks = (int)ceil_div(n, rpb);
    SCN_TRY(tmp.get((void **)&counts, sizeof(int) * (size_t)blocks * R));
    SCN_TRY(tmp.get((void **)&totals, sizeof(int) * (size_t)passes * R));
    SCN_CUDA_CHECK(cudaMemsetAsync(totals, 0, sizeof(int) * (size_t)passes * R, stream));
    if (passes > 1) {
      SCN_TRY(tmp.get((void **)&keys[1], sizeof(KEY) * (size_t)n));
      SCN_TRY(tmp.get((void **)&rows, sizeof(int) * (size_t)n));
    }
    // the row arrays alternate so that the last pass writes ord.order
    const int *src = nullptr;
    for (int p = 0; p < passes; ++p) {
      int *dst = ((passes - 1 - p) & 1) ? rows : ord.order;
      KEY *kin = keys[p & 1], *kout = p + 1 < passes ? keys[(p + 1) & 1] : nullptr;
      SCN_LAUNCH((k_order_count<KEY>), blocks, kCountThreads, 0, stream, kin, n, (int)rpb, p * digit, R, counts, totals + (size_t)p * R);
      SCN_LAUNCH((k_order_scatter<KEY>), blocks, kScatterThreads, 0, stream, kin, src, n, (int)rpb, p * digit, R, counts, totals + (size_t)p * R, kout, dst);
      src = dst;
    }
  }
  SCN_LAUNCH((k_order_tiles<WORDS>), (unsigned)ceil_div(ord.n_tiles * 32, 256), 256, 0, stream, ord.order, n, ord.n_tiles * kTile, masks, ord.tile_bits, ord.n_tiles);
  SCN_CUDA_CHECK(cudaGetLastError());
  return SCN_OK;
}

}  // namespace

void free_row_order(RowOrder &o, cudaStream_t stream) {
  device_free(o.order, stream);
  device_free(o.tile_bits, stream);
  o = RowOrder{};
}

// Builds the packing order of a rulebook table [K][n] if it is not there yet.
int rulebook_row_order(const Rulebook &rb, const int *table, long long n, RowOrder &ord, cudaStream_t stream) {
  if (ord.order || n == 0) return SCN_OK;
  const int K = rb.n_offsets;
  SCN_REQUIRE(K >= 1 && K <= kOrderMaxOffsets && n < (1ll << 31), SCN_ERR_UNSUPPORTED, "row order: %d offsets", K);
  KeyBits B;
  const int bits = key_bits(rb.dim, rb.filter, K, B);
  RowOrder o;
  o.words = K <= 32 ? 1 : 4;
  o.n_tiles = ceil_div(n, kTile);
  int st = device_alloc((void **)&o.order, sizeof(int) * (size_t)o.n_tiles * kTile, stream);
  if (st == SCN_OK) st = device_alloc((void **)&o.tile_bits, sizeof(unsigned) * (size_t)o.words * o.n_tiles, stream);
  // one tile per SM or fewer: nothing to gain from the order
  const bool sort = n >= 4096 && !(getenv("SCN_ROW_ORDER") && atoi(getenv("SCN_ROW_ORDER")) == 0);
  if (st == SCN_OK)
    st = K <= 32 ? build<unsigned, 1>(table, n, K, B, bits, o, sort, stream)
                 : build<unsigned long long, 4>(table, n, K, B, bits, o, sort, stream);
  if (st != SCN_OK) {
    free_row_order(o, stream);
    return st;
  }
  ord = o;
  return SCN_OK;
}

}  // namespace scn
