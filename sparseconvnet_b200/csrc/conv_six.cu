// fp32 sparse convolution on tcgen05 tensor cores over mask-sorted row tiles: results as accurate as fp32 multiply-adds.
//
// Same mathematics as the other convolution kernels (the reference's per-offset gather / GEMM / scatter-add is
// CPU/Convolution.cpp:137-148, CUDA/Convolution.cu:57-233), in the precision of k_conv_fma (conv_fma.cu):
//   * Every operand is written as the sum of three bf16 values, x = h + m + l: h = bf16(x), m = bf16(x - h), l = bf16(x - h - m).
//     The three hold the 24 bits of x exactly.  A product is the six terms h h', h m', m h', h l', m m', l h'.  With m up to
//     2^-8 of the value's power of two and l up to 2^-17, the two terms left out, m l' and l m', reach 2^-24 of a product at the
//     very worst, as much as rounding an fp32 product can take, and are some 2^-28 in the mean.
//   * The tensor core truncates its running sum, so it never runs far: one step of 32 planes of one filter offset is
//     summed there, the large terms and the small ones apart or the small ones first, and every step's sums are added to fp32
//     registers, rounded to nearest (the "drain" warps).
// Time and error against float64 beside k_conv_fma's: the table at conv_six_takes.
//
// The range of bf16 is that of fp32, so the low parts of a value near its lower end would be lost.  Rows and weights are split
// 2^24 times as large as they are and sums made 2^48 times smaller: then the last bit of the smallest fp32 value is a normal
// bf16 number, and the terms of a product are exact for every product that is a normal number, whatever stands beside it.
// Upwards that leaves less room, and an infinity has no low part: the pass that splits leaves the largest magnitude of rows and
// weights, and where a sum could overflow the kernel multiplies plain fp32 values instead (slow_items).  So it does where the
// largest products are near the lower end, where k_conv_fma's own rounding of subnormal sums is kept.
//
// Roles (19 or 15 warps, one CTA per SM, persistent), as in k_conv_tile but for the drain:
//   entries     one thread: a record per item, a slot per (tile, filter offset with a rule), 512 bytes of input rows from the table
//   producers   8 (4) warps, four to a step: 128 rows of 192 bytes ([32 h | 32 m] and [32 l]) by 16-byte cp.async; the first
//               lane of a step's warps orders its [W_h | W_m | W_l], one bulk copy
//   MMA         two warps; up to 64 output planes three instructions per 16 input planes, h (W_h | W_m | W_l), m (W_h | W_m), l W_h, into
//               three column ranges; above that six into one: the drain waits for what it reads beside the tensor core's own
//               traffic, 1 100 cycles per step of 96 planes with two ranges, more than the step's 700 of instructions
//   drain       8 warps, a row and half of the planes per lane: TMEM -> registers after every step, and after the tile's
//               last one through shared memory -> bias -> optional BatchNorm -> 16-byte stores, four lanes per row
// Tensor pipe active 74 % for 128 output planes, 54 for 96 (200 k rows, 1 050 and 1 070 cycles per step); below that no unit is near
// its peak: 64 planes 38 % beside 64 % of the issue slots and 1 030 cycles per step, 32 planes 22 and 60 %, 880 cycles.  As multiply-adds
// the same step is 1 024 to 4 096 cycles of the whole FMA pipe.  The barriers of the next step are looked at while this one is
// under way and the loads of a row's stores come before its branches: with a wait, a look at the abort flag and a role for the
// weights in every step, 200 k rows: 32 -> 32 planes 102 us, 89 now; 64 -> 64 229, 205; 96 -> 96 372, 318; 128 -> 128 525, 445; a
// Deconvolution 128 -> 96 to 43 k rows 28, 17.  (64 planes: three loads of 16 columns under one wait do not fit the registers, 216;
// two column ranges and with them four accumulators 204; sixteen drain warps 207.)  Rows split once per call, not once per gather:
// with fp32 rows (16 KB per step) split by the producers on their way through registers a step took twice as long.
//
// Every wait is bounded; on expiry the role raises the abort flag, everybody leaves, tensor memory is freed and
// the host sees FLAG_TC_TIMEOUT through scn_md_poll_errors.
#include <stdlib.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "conv_tile.cuh"

namespace scn {

namespace {

constexpr int kRows = kOrderTile;
constexpr int kDrainWarps = 8, kMmaWarps = 2;
constexpr int kSlots = 8;  // offsets the entries run ahead; even, so that a producing warp comes by every slot or every second
constexpr int kMaxStages = 12;
constexpr int kEpiBytes = 32 * 64;   // per drain warp: 32 rows x 16 planes on their way from lanes to whole lines
constexpr int kScale = 24;           // of rows and of weights, as a power of two
constexpr float kUp = 1 << kScale, kDown = 1.f / kUp / kUp;
constexpr int kRangeWords = 512;     // behind split rows and weight image: largest magnitude (float bits), one per block
constexpr int kPrepareThreads = 512, kPrepareBlocks = 296;

struct SixParams {
  const unsigned char *in_split;  // per row and slice of SP planes [SP h | SP m | SP l]
  const unsigned *in_range;
  long long row_bytes;
  long long n_in;
  float *out;  // n_split == 1: [n_out][cout]; else partial sums [n_split][n_tiles * 128][cout]
  int cout, cb, n_cb;  // output planes; planes of a column block (a multiple of 16, at most 128); column blocks
  const unsigned char *wprep;  // [K][column block][slice][h, m, l]
  const unsigned *w_range;
  const float *bias, *bn_scale, *bn_shift;
  float leak;
  const int *order, *packed, *by_work;
  const unsigned *tile_bits;
  int words;
  int K, n_slices, log2_terms;  // log2_terms: of the products of a sum, rounded up
  int n_stages;
  long long n_tiles, n_items;
  int n_split, per_tile;  // parts of a tile's offsets; items of a tile (parts x column blocks)
  // for slow_items: the operands as they are
  const float *in, *in_b, *weight, *pre_scale, *pre_shift;
  float pre_leak;
  int cin, planes_a;
  int drop;  // test hook: leave out one barrier arrival of the first CTA
  int *flags;
};

// Warps by role.  With 64 planes per drain lane (and weights that leave room for four stages) fewer producers, for
// 128 registers a thread.
template <int NA>
struct SixWarps {
  static constexpr int PROD = NA == 64 ? 4 : 8, GROUPS = PROD / kStepWarps;
  static constexpr int DRAIN0 = PROD, MMA = DRAIN0 + kDrainWarps, ENTRIES = MMA + kMmaWarps, THREADS = (ENTRIES < 15 ? 16 : ENTRIES + 1) * 32;  // (slow_items has 512 threads)
};

template <int SP>
struct SixShape {
  static constexpr unsigned HM = SP * 4, L = SP * 2;  // bytes of a row of a stage: [h | m], and [l]
  static constexpr unsigned A_BYTES = kRows * (HM + L);
  static constexpr int PIECES = HM / 16, NI = 32 / (32 / PIECES);  // 16-byte pieces per row, rows per lane (a warp has 32 rows)
  static constexpr int L_PIECES = L / 16, L_NI = 32 / (32 / L_PIECES);
  static_assert(NI == 2 * L_NI, "a lane's rows for [l] are half of those for [h | m]");
  static_assert(HM == 128 || HM == 64, "swizzled rows");
};

struct Ctl {
  unsigned long long full[kMaxStages], empty[kMaxStages];  // rows and weights landed; MMAs done
  unsigned long long s_full[kSlots], s_empty[kSlots], acc_full[4], acc_empty[4];
  unsigned long long r_full[kRecords], r_empty[kRecords];
  ItemRecord record[kRecords];  // part: the item within its tile
  int slot_k[kSlots];  // filter offset + (column block << 10); -1: no more work; + kNoRules: offset 0 with rows of zeros
  OrderedCopies ordered;
  unsigned tmem, range[2];
  int abort;
};

struct Item {
  long long tile;
  int part, block;
};
__device__ __forceinline__ Item item_at(const SixParams &P, long long item) {
  const int per = P.n_split * P.n_cb, rest = (int)(item % per);
  const long long i = item / per;
  return Item{P.by_work ? (long long)__ldg(P.by_work + i) : P.n_tiles - 1 - i, rest / P.n_cb, rest % P.n_cb};
}

// Where a row of an item's result goes.
__device__ __forceinline__ float *result_row(const SixParams &P, const Item &I, int position, int row) {
  return P.out + (P.n_split > 1 ? ((long long)I.part * P.n_tiles + I.tile) * kRows + position : (long long)row) * P.cout;
}

__device__ __forceinline__ float finished(const SixParams &P, float v, int c) {
  if (P.n_split > 1) return v;
  if (P.bias) v += __ldg(P.bias + c);
  if (P.bn_scale) {  // separate multiply and add, as the stand-alone BatchNorm kernel rounds them
    v = __fadd_rn(__fmul_rn(v, __ldg(P.bn_scale + c)), __ldg(P.bn_shift + c));
    v *= v > 0.f ? 1.f : P.leak;
  }
  return v;
}

// Operands whose parts bf16 cannot hold: infinities, NaN, products near either end of the range.  Plain fp32 multiply-adds in
// the order of k_conv_fma: the CTA's first 512 threads are four groups of 128, each with a tile and 32 of its planes, 8 x 4 results
// in registers per thread, and rows and weights of 32 input planes in one of two stages while the other is multiplied.  Layers on
// 200 k rows with one infinity, us here / on k_conv_fma: 32 -> 32 planes 297/190, 64 -> 64 977/574, 96 -> 96 1 818/1 478, 160 -> 160
// 5 720/3 990; with a warp per row and a lane per plane, which reuses no weight, 5 580 to 62 600.  What it costs the layers
// that do not come here decided its form: inlined, with 8 x 8 results, with eight rows per warp and no shared memory, or as a
// kernel of its own behind every k_conv_six it took 1 to 3 % of their time; as a call across which nothing lives, none.
constexpr int kFmaGroup = 128, kFmaGroups = 4, kFmaChunk = 32;  // threads of a group; input planes of a step
constexpr int kFmaPlanes = 32, kFmaX = kFmaPlanes / 4, kFmaY = kFmaGroup / kFmaX, kFmaRows = kRows / kFmaY;
constexpr int kFmaRing = 4;                                       // offsets whose entries are there
constexpr int kFmaStride = kFmaChunk + 4;                         // floats of a row of a stage: broadcast loads on different banks
constexpr int kFmaStage = kRows * kFmaStride + kFmaChunk * kFmaPlanes;  // floats: rows, weights
constexpr int kFmaShare = 2 * kFmaStage + kFmaRing * kRows;
// the threads of one group
__device__ __forceinline__ void group_sync(int group) {
  if (group == 0) asm volatile("bar.sync 1, %0;" ::"n"(kFmaGroup) : "memory");
  else if (group == 1) asm volatile("bar.sync 2, %0;" ::"n"(kFmaGroup) : "memory");
  else if (group == 2) asm volatile("bar.sync 3, %0;" ::"n"(kFmaGroup) : "memory");
  else asm volatile("bar.sync 4, %0;" ::"n"(kFmaGroup) : "memory");
}

// one group's share (n0: its first plane in the column block) of an item
__device__ __forceinline__ void slow_item(const SixParams &P, long long item, int n0, float *stages, bool finite_weights) {
  constexpr int BN = kFmaPlanes, TM = kFmaRows;
  const int tid = threadIdx.x % kFmaGroup, group = threadIdx.x / kFmaGroup;
  const Item I = item_at(P, item);
  const int last_plane = min(P.cb, P.cout - I.block * P.cb) - n0;  // planes of the share, counted from n0
  n0 += I.block * P.cb;
  unsigned m[4];
#pragma unroll
  for (int w = 0; w < 4; ++w) m[w] = w < P.words ? __ldg(P.tile_bits + I.tile * P.words + w) : 0u;
  const int total = __popc(m[0]) + __popc(m[1]) + __popc(m[2]) + __popc(m[3]), first = total * I.part / P.n_split;
  const int last = total * (I.part + 1) / P.n_split;
  if (P.n_split > 1) keep_range(m, first, last);
  const int nch = (P.cin + kFmaChunk - 1) / kFmaChunk;
  const int tx = tid % kFmaX, ty = tid / kFmaX;
  static_assert(kRows == kFmaGroup, "a thread per entry");
  int *ring = reinterpret_cast<int *>(stages + 2 * kFmaStage);
  const int *packed = P.packed + (I.tile * P.K + first) * kRows + tid;
  const int offsets = last - first;
  for (int o = 0; o < min(2, offsets); ++o) ring[o * kRows + tid] = __ldg(packed + o * kRows);
  group_sync(group);

  // copying: eight threads per row, 16 rows at a time; a thread per 16 bytes of weights
  constexpr int CR = kFmaGroup / 8, CI = kRows / CR, WP = BN / 4, WR = kFmaGroup / WP;
  const int cj = (tid & 7) * 4, cr = tid >> 3, wc = tid % WP * 4, wr = tid / WP;
  int k_issue = 0, c_issue = 0, o_issue = 0;  // filter offset, chunk and offset of the item of the step to be issued next
  auto issue = [&](int s) {                   // one cp.async group per call, empty past the end
    if (o_issue < offsets) {
      if (c_issue == 0) {  // the lowest offset of those that are left
#pragma unroll
        for (int w = 3; w >= 0; --w)
          if (m[w]) k_issue = w * 32 + __ffs(m[w]) - 1;
#pragma unroll
        for (int w = 0; w < 4; ++w)
          if (w == k_issue >> 5) m[w] &= m[w] - 1;
        if (o_issue + 2 < offsets)  // the entries of the offset after the next: here when they are asked for
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(ring + ((o_issue + 2) % kFmaRing) * kRows + tid)), "l"(packed + (o_issue + 2) * kRows) : "memory");
      }
      float *a = stages + (s & 1) * kFmaStage, *w = a + kRows * kFmaStride;
      const int c = c_issue * kFmaChunk + cj;
      if (c < P.cin) {
        const float *src = !P.in_b ? P.in + c : c < P.planes_a ? P.in + c : P.in_b + (c - P.planes_a);
        const int ld = !P.in_b ? P.cin : c < P.planes_a ? P.planes_a : P.cin - P.planes_a;
        const int *entry = ring + o_issue % kFmaRing * kRows + cr;
#pragma unroll
        for (int i = 0; i < CI; ++i) {
          const int v = entry[i * CR];
          const bool hit = (unsigned)v < (unsigned)P.n_in;
          if (v >= 0 && !hit) atomicOr(P.flags, FLAG_BAD_ROW);
          cp_async16(smem_u32(a + (cr + i * CR) * kFmaStride + cj), hit ? src + (long long)v * ld : P.in, hit ? 16u : 0u);
        }
      }
      const float *wk = P.weight + ((long long)k_issue * P.cin + c_issue * kFmaChunk) * P.cout + n0 + wc;
      const int rows = min(kFmaChunk, P.cin - c_issue * kFmaChunk);
#pragma unroll
      for (int i = 0; i < kFmaChunk / WR; ++i) {
        const int r = wr + i * WR;
        const bool ok = r < rows && wc < last_plane;
        cp_async16(smem_u32(w + r * BN + wc), ok ? wk + (long long)r * P.cout : P.weight, ok ? 16u : 0u);
      }
      if (++c_issue == nch) c_issue = 0, ++o_issue;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float acc[TM][4];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
  issue(0);
  issue(1);
  int chunk = 0, o = 0;
  const int steps = offsets * nch;
  for (int s = 0; s < steps; ++s) {
    float *a = stages + (s & 1) * kFmaStage;
    const float *w = a + kRows * kFmaStride + tx * 4;
    const int *entry = ring + o % kFmaRing * kRows;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    if (P.pre_scale && chunk * kFmaChunk + cj < P.cin) {  // the pieces that this thread has copied, rounded as in k_six_prepare
      const int c = chunk * kFmaChunk + cj;
#pragma unroll 1
      for (int i = 0; i < CI; ++i)
        if ((unsigned)entry[cr + i * CR] < (unsigned)P.n_in) {
          float *x = a + (cr + i * CR) * kFmaStride + cj;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float y = __fadd_rn(__fmul_rn(x[e], __ldg(P.pre_scale + c + e)), __ldg(P.pre_shift + c + e));
            x[e] = y * (y > 0.f ? 1.f : P.pre_leak);
          }
        }
    }
    group_sync(group);
    const int kmax = min(kFmaChunk, P.cin - chunk * kFmaChunk);
    a += ty * kFmaStride;
    // A row without a rule counts as zeros, but is no business of an infinite weight.
    auto multiply = [&](auto all) {
#pragma unroll 1
      for (int kk = 0; kk < kmax; kk += 4) {
        float4 wv[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) wv[q] = *reinterpret_cast<const float4 *>(w + (kk + q) * BN);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          if (!decltype(all)::value && (unsigned)entry[ty + i * kFmaY] >= (unsigned)P.n_in) continue;
          const float4 av = *reinterpret_cast<const float4 *>(a + i * kFmaY * kFmaStride + kk);
          const float x[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            acc[i][0] = fmaf(x[q], wv[q].x, acc[i][0]);
            acc[i][1] = fmaf(x[q], wv[q].y, acc[i][1]);
            acc[i][2] = fmaf(x[q], wv[q].z, acc[i][2]);
            acc[i][3] = fmaf(x[q], wv[q].w, acc[i][3]);
          }
        }
      }
    };
    if (finite_weights) multiply(std::true_type());
    else multiply(std::false_type());
    if (++chunk == nch) chunk = 0, ++o;
    group_sync(group);
    issue(s + 2);
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int p = ty + i * kFmaY, row = __ldg(P.order + I.tile * kRows + p);
    if (row < 0) continue;
    float *to = result_row(P, I, p, row) + n0 + tx * 4;
    if (tx * 4 < last_plane)
#pragma unroll
      for (int e = 0; e < 4; ++e) to[e] = finished(P, acc[i][e], n0 + tx * 4 + e);
  }
}

// all items of a CTA, by its first 512 threads
__device__ __noinline__ void slow_items(const SixParams &P, float *smem, bool finite_weights) {
  const int group = threadIdx.x / kFmaGroup, cols = (P.cb + kFmaPlanes - 1) / kFmaPlanes;
  const long long n = items_here(P.n_items) * cols;
  for (long long u = group; u < n; u += kFmaGroups)
    slow_item(P, item_of(u / cols), (int)(u % cols) * kFmaPlanes, smem + group * kFmaShare, finite_weights);
}

// Can sums of 2^log2_terms products of values up to x and w in magnitude (float bits) be made of bf16 parts?  Nothing may
// reach infinity on the way.
__device__ __forceinline__ bool parts_reach(unsigned x, unsigned w, int log2_terms) {
  const int ex = (int)(x >> 23) - 127, ew = (int)(w >> 23) - 127;  // (128: infinity or NaN)
  if (ex + kScale >= 126 || ew + kScale >= 126) return false;
  if (x == 0 || w == 0) return true;
  return ex >= -60 && ew >= -60 && ex + ew >= -90 && ex + ew + 2 * kScale + 2 + log2_terms < 126;
}

// 2^24 x = h + m + l, two values at a time (the first in the low half)
__device__ __forceinline__ void split3_pair(float a, float b, unsigned &h, unsigned &m, unsigned &l) {
  a *= kUp, b *= kUp;
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  h = *reinterpret_cast<unsigned *>(&v);
  const float a1 = a - __uint_as_float(h << 16), b1 = b - __uint_as_float(h & 0xFFFF0000u);
  v = __floats2bfloat162_rn(a1, b1);
  m = *reinterpret_cast<unsigned *>(&v);
  v = __floats2bfloat162_rn(a1 - __uint_as_float(m << 16), b1 - __uint_as_float(m & 0xFFFF0000u));
  l = *reinterpret_cast<unsigned *>(&v);
}

// SP: input planes of a step; NA: planes of a drain warp, a multiple of 16
template <int SP, int NA>
__global__ void __launch_bounds__(SixWarps<NA>::THREADS, 1) k_conv_six(const __grid_constant__ SixParams P) {
  SCN_GRID_WAIT();
  using Shape = SixShape<SP>;
  using Warps = SixWarps<NA>;
  constexpr int kProdWarps = Warps::PROD, kDrain0 = Warps::DRAIN0, kMma = Warps::MMA, kEntries = Warps::ENTRIES, kProdGroups = Warps::GROUPS;
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned w_part = (unsigned)P.cb * SP * 2, w_bytes = w_part * 3;
  const unsigned stage_bytes = Shape::A_BYTES + ((w_bytes + 1023u) & ~1023u);  // the swizzle pattern repeats every 1 KB
  const unsigned smem0 = smem_u32(smem);
  unsigned char *tail = smem + (size_t)P.n_stages * stage_bytes;
  int *entries = reinterpret_cast<int *>(tail);  // [kSlots][128] input row of every tile row, or -1
  unsigned char *epi = tail + sizeof(int) * kSlots * kRows;
  Ctl &C = *reinterpret_cast<Ctl *>(epi + kDrainWarps * kEpiBytes);
  constexpr bool kJoint = NA <= 32;             // (up to 64 planes) [W_h | W_m | W_l] as one operand, a range of columns for each
  constexpr int kGroup = kJoint ? 32 / SP : 1;  // steps summed in tensor memory before they are drained
  const int dcols = ((kJoint ? 3 : 1) * P.cb + 31) & ~31;
  const int n_acc = min(4, 512 / dcols) & ~1;  // (an accumulator belongs to one of the issuing warps)
  const long long my_items = items_here(P.n_items);  // (the grid has at most n_items CTAs)

  if (tid < 2) C.range[tid] = 0;
  if (tid == 0) {
    for (int i = 0; i < P.n_stages; ++i) {
      mbar_init(&C.full[i], kStepWarps * 32 + 1);  // the lanes of the producing warps, and the weights
      mbar_init(&C.empty[i], kMmaWarps);
    }
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&C.s_full[i], 1);
      mbar_init(&C.s_empty[i], kStepWarps * min(P.n_slices, kProdGroups));  // the producing warps that come by
    }
    for (int i = 0; i < kRecords; ++i) {
      mbar_init(&C.r_full[i], 1);
      mbar_init(&C.r_empty[i], kDrainWarps + kMmaWarps);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&C.acc_full[i], 1);
      mbar_init(&C.acc_empty[i], kDrainWarps);
    }
    C.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  static_assert(Warps::THREADS >= kRangeWords, "a thread per range word");
  if (tid < kRangeWords) {
    const unsigned x = __reduce_max_sync(0xffffffffu, __ldg(P.in_range + tid)), w = __reduce_max_sync(0xffffffffu, __ldg(P.w_range + tid));
    if (lane == 0) atomicMax(&C.range[0], x), atomicMax(&C.range[1], w);
  }
  if (warp == kMma) tmem_alloc(&C.tmem, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = C.tmem;
  volatile int *abort = &C.abort;

  if (!parts_reach(C.range[0], C.range[1], P.log2_terms)) {
    if (tid < kFmaGroups * kFmaGroup) slow_items(P, reinterpret_cast<float *>(smem), C.range[1] < 0x7F800000u);
    __syncthreads();
    if (threadIdx.x >> 5 == kMma) tmem_dealloc(C.tmem, 512);
    return;
  }
  if (warp < kProdWarps) {
    // ==================================== producers =============================================
    // Group g of four warps takes the steps g, g + kProdGroups, ...; a warp copies 32 rows of a step, a lane one 16-byte piece of
    // [h | m] of the rows q NI .. q NI + NI - 1 of them and one of [l] of half of these.  The input rows of the next step are in
    // registers before its stage is free.  A warp leaves as a whole: what its lanes do together has no limit to its wait for one
    // that has gone.
    const int j = lane % Shape::PIECES, q = lane / Shape::PIECES, lj = lane % Shape::L_PIECES, lq = lane / Shape::L_PIECES;
    const int group = warp / kStepWarps, row0 = warp % kStepWarps * 32 + q * Shape::NI, l_row0 = warp % kStepWarps * 32 + lq * Shape::L_NI;
    // (where a 16-byte chunk c of row r goes: rows_desc; rows of 128 bytes come in eights, of 64 in fours, of 32 in twos)
    const unsigned hm_dst = smem0 + (unsigned)row0 * Shape::HM + (unsigned)((Shape::HM == 128 ? j : j ^ (q & 1) * 2) * 16);
    const unsigned l_dst = smem0 + kRows * Shape::HM + (unsigned)l_row0 * Shape::L +
                           (unsigned)((Shape::L == 64 ? lj ^ (lq & 1) * 2 : lj ^ (lq >> 1 & 1)) * 16);
    const int d_slot = kProdGroups / P.n_slices, d_slice = kProdGroups % P.n_slices;
    int slot = group / P.n_slices, slice = group % P.n_slices, st = group, par = 1;  // (n_stages is at least kProdGroups)
    const bool brings_weights = warp % kStepWarps == 0 && lane == 0;
    int slot_k = 0, filled = 0;
    bool ok = true, bad = false, fresh = true;
    int rows[Shape::NI];
    for (;;) {
      if (fresh) {
        const int si = slot % kSlots;
        // (A warp comes by every slot, or by every second one with one slice: it has seen the slot kSlots before this one
        // filled, so the parity cannot be that of an earlier round.)
        ok = mbar_wait_warp(&C.s_full[si], (slot / kSlots) & 1, abort);
        if (!ok) break;
        slot_k = C.slot_k[si];
        if (slot_k < 0) break;
        const int *ent = entries + si * kRows + row0;
#pragma unroll
        for (int i = 0; i < Shape::NI; i += 4) {
          const int4 e4 = *reinterpret_cast<const int4 *>(ent + i);
          rows[i] = e4.x, rows[i + 1] = e4.y, rows[i + 2] = e4.z, rows[i + 3] = e4.w;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&C.s_empty[si]);
#pragma unroll
        for (int i = 0; i < Shape::NI; ++i) {
          if (slot_k >= kNoRules) rows[i] = -1;
          bad |= rows[i] >= (int)P.n_in;
        }
      }
      ok = mbar_wait_warp(&C.empty[st], par, abort);  // (the first round passes)
      if (!ok) break;
      const unsigned at = (unsigned)st * stage_bytes;
      if (brings_weights && !(P.drop && blockIdx.x == 0 && group == 0 && filled == 0)) {
        const int k = slot_k & 1023, block = slot_k >> 10 & 1;
        mbar_expect_tx(&C.full[st], w_bytes);
        bulk_copy_g2s(smem0 + at + Shape::A_BYTES, P.wprep + ((size_t)(k * P.n_cb + block) * P.n_slices + slice) * w_bytes, w_bytes, &C.full[st]);
      }
      ++filled;
      const unsigned char *col = P.in_split + slice * (SP * 6) + j * 16, *l_col = P.in_split + slice * (SP * 6) + SP * 4 + lj * 16;
#pragma unroll
      for (int i = 0; i < Shape::NI; ++i) {
        const bool hit = (unsigned)rows[i] < (unsigned)P.n_in;
        const unsigned swizzle = (Shape::HM == 128 ? i & 7 : i >> 1 & 3) * 16;
        cp_async16(((hm_dst + at) ^ swizzle) + i * Shape::HM, col + (size_t)(unsigned)(hit ? rows[i] : 0) * P.row_bytes, hit ? 16u : 0u);
      }
#pragma unroll
      for (int i = 0; i < Shape::L_NI; ++i) {
        const int row = lq & 1 ? rows[Shape::L_NI + i] : rows[i];
        const bool hit = (unsigned)row < (unsigned)P.n_in;
        const unsigned swizzle = (Shape::L == 64 ? i >> 1 & 3 : i >> 2 & 1) * 16;
        cp_async16(((l_dst + at) ^ swizzle) + i * Shape::L, l_col + (size_t)(unsigned)(hit ? row : 0) * P.row_bytes, hit ? 16u : 0u);
      }
      cp_async_arrive(&C.full[st]);
      slot += d_slot, slice += d_slice;
      fresh = d_slot > 0;
      if (slice >= P.n_slices) slice -= P.n_slices, ++slot, fresh = true;
      st += kProdGroups;
      if (st >= P.n_stages) st -= P.n_stages, par ^= 1;
    }
    if (bad) atomicOr(P.flags, FLAG_BAD_ROW);
    asm volatile("cp.async.wait_all;" ::: "memory");  // they must land before the CTA's shared memory goes away
    if (brings_weights) C.ordered.slabs[group] = filled;
    if (!ok) *abort = 1;
  } else if (warp < kMma + kMmaWarps && warp >= kMma) {
    // ==================================== MMA issue =============================================
    // Two warps take the accumulators in turn: what one spends on barriers passes while the other's instructions run (U-Net
    // of two rooms 2 985 -> 2 950 us).  The whole warp runs the loop and one elected lane issues, by a predicate (mma_bf16_if).
    const unsigned id1 = tile_idesc(P.cb), id2 = tile_idesc(kJoint ? 2 * P.cb : 16), id3 = tile_idesc(kJoint ? 3 * P.cb : 16);
    const unsigned long long a_desc = rows_desc<Shape::HM>(smem0, 0), l_desc = rows_desc<Shape::L>(smem0, kRows * Shape::HM);
    const unsigned long long w_desc = smem_desc(smem0 + Shape::A_BYTES, 128, SP / 8 * 128);
    const unsigned a_hi = (unsigned)(a_desc >> 32), l_hi = (unsigned)(l_desc >> 32), w_hi = (unsigned)(w_desc >> 32);
    const unsigned a0 = (unsigned)a_desc, l0 = (unsigned)l_desc, w0 = (unsigned)w_desc;
    const unsigned stage_step = stage_bytes >> 4, wm_step = w_part >> 4;
    const int items = (int)my_items, n_stages = P.n_stages, cb = P.cb;
    int st = 0, par = 0, buf = 0, buf_par = 1;
    unsigned d = tmem;
    bool ok = true;
    const unsigned lead = elect_one() ? 1u : 0u;
    bool mine = warp == kMma;  // the next accumulator is this warp's
    bool ready = false, acc_ready = false;  // the stage and the accumulator at hand, looked at a step earlier
    for (int i = 0; i < items && ok; ++i) {
      const int ri = i % kRecords;
      if (!mbar_wait_warp(&C.r_full[ri], (i / kRecords) & 1)) {
        ok = false;
        break;
      }
      const int steps = __reduce_max_sync(0xffffffffu, C.record[ri].steps);
      if (lead) mbar_arrive(&C.r_empty[ri]);
      for (int s = 0; s < steps; ++s) {
        const bool opens = s % kGroup == 0, closes = s % kGroup == kGroup - 1 || s == steps - 1;
        // the accumulator must have been drained
        if (opens && mine && !acc_ready && (__any_sync(0xffffffffu, *abort != 0) || !mbar_wait_warp(&C.acc_empty[buf], buf_par))) {
          ok = false;
          break;
        }
        if (!ready && !mbar_wait_warp(&C.full[st], par)) {
          ok = false;
          break;
        }
        const int st1 = st + 1 == n_stages ? 0 : st + 1, par1 = st1 ? par : par ^ 1;
        const int buf1 = !closes ? buf : buf + 1 == n_acc ? 0 : buf + 1, buf_par1 = closes && buf1 == 0 ? buf_par ^ 1 : buf_par;
        const unsigned seen = mbar_test(&C.full[st1], par1), acc_seen = mbar_test(&C.acc_empty[buf1], buf_par1);
        // (the other warp's steps too, and a stage goes when both have been here: neither can fall a round behind, or run a round
        // ahead, where a phase's parity is that of another)
        if (!mine) {
          if (lead) mbar_arrive(&C.empty[st]);
        } else {
          // order the copied rows (acquired through the barrier) before the tensor core's async-proxy reads
          fence_proxy_async_smem();
          tc_fence_after();
          const unsigned at = (unsigned)st * stage_step;
          if (kJoint) {
#pragma unroll
            for (int jj = 0; jj < SP / 16; ++jj) {
              const unsigned ah = a0 + at + jj * 2, am = ah + SP / 8, al = l0 + at + jj * 2, wh = w0 + at + jj * 16;
              if (jj == 0) mma_bf16_if(lead, d, ah, a_hi, wh, w_hi, id3, opens ? 0u : 1u);
              else mma_bf16_acc_if(lead, d, ah, a_hi, wh, w_hi, id3);
              mma_bf16_acc_if(lead, d + cb, am, a_hi, wh, w_hi, id2);
              mma_bf16_acc_if(lead, d + 2 * cb, al, l_hi, wh, w_hi, id1);
            }
          } else {
            const unsigned wm = wm_step, wl = 2 * wm_step;
#pragma unroll
            for (int jj = 0; jj < SP / 16; ++jj) {  // 2^-16 of a product, 2^-8, then the large ones
              const unsigned ah = a0 + at + jj * 2, am = ah + SP / 8, al = l0 + at + jj * 2, wh = w0 + at + jj * 16;
              if (jj == 0) mma_bf16_if(lead, d, al, l_hi, wh, w_hi, id1, 0u);
              else mma_bf16_acc_if(lead, d, al, l_hi, wh, w_hi, id1);
              mma_bf16_acc_if(lead, d, ah, a_hi, wh + wl, w_hi, id1);
              mma_bf16_acc_if(lead, d, am, a_hi, wh + wm, w_hi, id1);
            }
#pragma unroll
            for (int jj = 0; jj < SP / 16; ++jj) {
              const unsigned ah = a0 + at + jj * 2, am = ah + SP / 8, wh = w0 + at + jj * 16;
              mma_bf16_acc_if(lead, d, am, a_hi, wh, w_hi, id1);
              mma_bf16_acc_if(lead, d, ah, a_hi, wh + wm, w_hi, id1);
            }
#pragma unroll
            for (int jj = 0; jj < SP / 16; ++jj) mma_bf16_acc_if(lead, d, a0 + at + jj * 2, a_hi, w0 + at + jj * 16, w_hi, id1);
          }
          tc_commit_if(lead, &C.empty[st]);
          if (closes) tc_commit_if(lead, &C.acc_full[buf]);
        }
        st = st1, par = par1;
        ready = __all_sync(0xffffffffu, seen != 0), acc_ready = __all_sync(0xffffffffu, acc_seen != 0);
        if (closes) mine = !mine;
        buf = buf1, buf_par = buf_par1, d = tmem + (unsigned)(buf * dcols);
      }
    }
    if (!ok) *abort = 1;
  } else if (warp == kEntries) {
    // ==================================== entries ===============================================
    if (lane == 0) {
      int slot = 0;
      bool ok = true;
      Tiles<SixParams> tiles;
      tiles.start(P);
      for (long long it = 0; it < my_items && ok; ++it) {
        unsigned u[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) u[w] = tiles.mask[w];
        const int tile = tiles.tile, within = P.per_tile == 1 ? 0 : (int)item_of(it) % P.per_tile, part = within / P.n_cb, block = within - part * P.n_cb;
        const int *src = P.packed + (long long)tile * P.K * kRows;
        tiles.advance(P, it);
        int offsets = __popc(u[0]) + __popc(u[1]) + __popc(u[2]) + __popc(u[3]);
        if (P.n_split > 1) {
          const int first = offsets * part / P.n_split, last = offsets * (part + 1) / P.n_split;
          keep_range(u, first, last);
          src += first * kRows;
          offsets = last - first;
        }
        // a tile (or part) without any rule still gets one step, of weights and rows of zeros
        const bool none = offsets == 0;
        if (none) u[0] = 1u;
        const int ri = (int)it % kRecords;
        if (!mbar_wait(&C.r_empty[ri], (((int)it / kRecords) + 1) & 1)) {
          ok = false;
          break;
        }
        C.record[ri] = ItemRecord{max(1, offsets) * P.n_slices, tile, within, tiles.tile};
        mbar_arrive(&C.r_full[ri]);
#pragma unroll 1
        for (int w = 0; w < 4 && ok; ++w) {
          unsigned m = u[0];
          u[0] = u[1], u[1] = u[2], u[2] = u[3], u[3] = 0;
          for (; m; m &= m - 1, ++slot, src += kRows) {
            const int si = slot % kSlots;
            if (!mbar_wait(&C.s_empty[si], ((slot / kSlots) + 1) & 1) || *abort) {
              ok = false;
              break;
            }
            C.slot_k[si] = (none ? kNoRules : w * 32 + __ffs(m) - 1) + (block << 10);
            if (none) {
              mbar_arrive(&C.s_full[si]);
            } else {
              mbar_expect_tx(&C.s_full[si], kRows * 4);
              bulk_copy_g2s(smem_u32(entries + si * kRows), src, kRows * 4, &C.s_full[si]);
            }
          }
        }
      }
      // every producing warp finds its next step in a slot that ends it
      const int ends = (kProdGroups - 1) / P.n_slices + 1;
      for (int i = 0; i < ends && ok; ++i, ++slot) {
        const int si = slot % kSlots;
        if (!mbar_wait(&C.s_empty[si], ((slot / kSlots) + 1) & 1)) {
          ok = false;
          break;
        }
        C.slot_k[si] = -1;
        mbar_arrive(&C.s_full[si]);
      }
      C.ordered.slots = slot;
      if (!ok) *abort = 1;
    }
  } else if (warp < kMma) {
    // ==================================== drain =================================================
    const int quad = warp & 3, half = (warp - kDrain0) >> 2;
    const int units = P.cb / 16, first_unit = half ? (units + 1) / 2 : 0, my_units = half ? units / 2 : (units + 1) / 2;
    float4 *my_epi = reinterpret_cast<float4 *>(epi + (warp - kDrain0) * kEpiBytes);
    const unsigned base0 = tmem + ((unsigned)(quad * 32) << 16) + (unsigned)(first_unit * 16);
    const int nc = P.cout, cb = P.cb;
    int buf = 0, buf_par = 0;
    bool ok = true;
    int next_orow = 0;  // this lane's row of the next item: asked for an item ahead
    bool ready = false;  // the accumulator at hand, looked at while the one before it was read
    for (int it = 0; it < (int)my_items && ok; ++it) {
      const int ri = it % kRecords;
      if (!mbar_wait_warp(&C.r_full[ri], (it / kRecords) & 1)) {
        ok = false;
        break;
      }
      const ItemRecord R = C.record[ri];
      __syncwarp();
      if (lane == 0) mbar_arrive(&C.r_empty[ri]);
      const int groups = (__reduce_max_sync(0xffffffffu, R.steps) + kGroup - 1) / kGroup;
      const Item I{R.tile, R.part / P.n_cb, R.part % P.n_cb};
      const int orow = it ? next_orow : __ldg(P.order + I.tile * kRows + quad * 32 + lane);
      next_orow = __ldg(P.order + (long long)R.next_tile * kRows + quad * 32 + lane);
      float acc[NA];
#pragma unroll
      for (int e = 0; e < NA; ++e) acc[e] = 0.f;
      for (int s = 0; s < groups; ++s) {
        if (!ready && (__any_sync(0xffffffffu, *abort != 0) || !mbar_wait_warp(&C.acc_full[buf], buf_par))) {
          ok = false;
          break;
        }
        tc_fence_after();
        const unsigned base = base0 + (unsigned)(buf * dcols);
#pragma unroll
        for (int u = 0; u < NA / 16; ++u)
          if (u < my_units) {
            if (!kJoint) {
              unsigned a[16];
              tmem_ld16_nowait(base + u * 16, a);
              tmem_wait_ld();
#pragma unroll
              for (int e = 0; e < 16; ++e) acc[u * 16 + e] += __uint_as_float(a[e]);
            } else {
#pragma unroll
              for (int e0 = 0; e0 < 16; e0 += 8) {
                unsigned a[8], b[8], c[8];
                tmem_ld8_nowait(base + u * 16 + e0, a);
                tmem_ld8_nowait(base + cb + u * 16 + e0, b);
                tmem_ld8_nowait(base + 2 * cb + u * 16 + e0, c);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 8; ++e)
                  acc[u * 16 + e0 + e] += __uint_as_float(a[e]) + (__uint_as_float(b[e]) + __uint_as_float(c[e]));
              }
            }
          }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&C.acc_empty[buf]);
        if (++buf == n_acc) buf = 0, buf_par ^= 1;
        ready = __all_sync(0xffffffffu, mbar_test(&C.acc_full[buf], buf_par) != 0);
      }
      if (!ok) break;
      // where rows lane / 4, + 8, + 16, + 24 of the warp go
      int to[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        to[i] = __shfl_sync(0xffffffffu, orow, i * 8 + (lane >> 2));
        if (P.n_split > 1 && to[i] >= 0) to[i] = (I.part * (int)P.n_tiles + R.tile) * kRows + quad * 32 + i * 8 + (lane >> 2);
      }
#pragma unroll
      for (int u = 0; u < NA / 16; ++u)
        if (u < my_units) {
#pragma unroll
          for (int e = 0; e < 16; e += 4)
            my_epi[lane * 4 + ((e >> 2) ^ ((lane >> 1) & 3))] = make_float4(acc[u * 16 + e] * kDown, acc[u * 16 + e + 1] * kDown, acc[u * 16 + e + 2] * kDown, acc[u * 16 + e + 3] * kDown);
          __syncwarp();
          const int c = I.block * cb + (first_unit + u) * 16 + (lane & 3) * 4;
          if (c < nc) {
            const bool finish = P.n_split == 1;
            float4 bias = make_float4(0.f, 0.f, 0.f, 0.f), sc = bias, sh = bias, v[4];
            if (finish && P.bias) bias = __ldg(reinterpret_cast<const float4 *>(P.bias + c));
            if (finish && P.bn_scale) {
              sc = make_float4(__ldg(P.bn_scale + c), __ldg(P.bn_scale + c + 1), __ldg(P.bn_scale + c + 2), __ldg(P.bn_scale + c + 3));
              sh = make_float4(__ldg(P.bn_shift + c), __ldg(P.bn_shift + c + 1), __ldg(P.bn_shift + c + 2), __ldg(P.bn_shift + c + 3));
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int row = i * 8 + (lane >> 2);
              v[i] = my_epi[row * 4 + ((lane & 3) ^ ((row >> 1) & 3))];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float *y = &v[i].x;
              if (finish && P.bias) v[i].x += bias.x, v[i].y += bias.y, v[i].z += bias.z, v[i].w += bias.w;
              if (finish && P.bn_scale) {  // separate multiply and add, as the stand-alone BatchNorm kernel rounds them
                v[i].x = __fadd_rn(__fmul_rn(v[i].x, sc.x), sh.x), v[i].y = __fadd_rn(__fmul_rn(v[i].y, sc.y), sh.y);
                v[i].z = __fadd_rn(__fmul_rn(v[i].z, sc.z), sh.z), v[i].w = __fadd_rn(__fmul_rn(v[i].w, sc.w), sh.w);
#pragma unroll
                for (int e = 0; e < 4; ++e) y[e] *= y[e] > 0.f ? 1.f : P.leak;
              }
              if (to[i] >= 0) *reinterpret_cast<float4 *>(P.out + to[i] * (long long)nc + c) = v[i];
            }
          }
          __syncwarp();
        }
    }
    if (!ok) *abort = 1;
  }
  tc_fence_before();
  __syncthreads();
  if (*abort) {
    if (tid == 0) atomicOr(P.flags, FLAG_TC_TIMEOUT);
    land_copies(C, P.n_stages, kProdGroups);
  }
  __syncwarp();
  if (warp == kMma) tmem_dealloc(tmem, 512);
}

struct PrepareParams {
  const float *in, *in_b;  // [n][cin], or the column-wise concatenation [in (planes_a) | in_b]
  unsigned char *rows;
  unsigned *in_range;
  long long n_pieces;      // of eight planes
  int cin, ppr, planes_a;
  const float *pre_scale, *pre_shift;
  float pre_leak;
  const float *weight;
  unsigned char *image;
  unsigned *w_range;
  long long w_pieces;
  int cout, cb, n_cb, n_slices;
  int row_blocks;          // the first blocks split rows, the others weights
};

__device__ __forceinline__ void split3_eight(const float (&x)[8], unsigned char *to, size_t part) {
  uint4 h, m, l;
  split3_pair(x[0], x[1], h.x, m.x, l.x);
  split3_pair(x[2], x[3], h.y, m.y, l.y);
  split3_pair(x[4], x[5], h.z, m.z, l.z);
  split3_pair(x[6], x[7], h.w, m.w, l.w);
  *reinterpret_cast<uint4 *>(to) = h;
  *reinterpret_cast<uint4 *>(to + part) = m;
  *reinterpret_cast<uint4 *>(to + 2 * part) = l;
}

// The operands of a layer as three bf16 parts, in one launch, and the largest magnitude of each (range words):
// rows     [n][cin] (or a join), optionally behind an eval-mode BatchNorm -> per row and slice of SP planes [SP h | SP m | SP l],
//          planes past cin zero; eight planes per thread and turn.  Bound by HBM: 32 bytes in, 48 out.
// weights  [K][cin][cout] -> [K][column block][slice][h, m, l][cb x SP] in the K-major core-matrix layout of the MMA's B operand,
//          eight input planes of an output plane per thread and turn.  Made anew in every call: nothing in this mode is computed
//          with weights of an earlier one.
template <int SP>
__global__ void __launch_bounds__(kPrepareThreads) k_six_prepare(PrepareParams P) {
  SCN_GRID_WAIT();
  const bool rows = (int)blockIdx.x < P.row_blocks;
  const int block = rows ? blockIdx.x : blockIdx.x - P.row_blocks, blocks = rows ? P.row_blocks : gridDim.x - P.row_blocks;
  const long long total = rows ? P.n_pieces : P.w_pieces;
  unsigned most = 0;
  for (long long idx = (long long)block * kPrepareThreads + threadIdx.x; idx < total; idx += (long long)blocks * kPrepareThreads) {
    float x[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = 0.f;
    if (rows) {
      const long long row = idx / P.ppr;
      const int c = (int)(idx - row * P.ppr) * 8;
#pragma unroll
      for (int half = 0; half < 8; half += 4)
        if (c + half < P.cin) {
          const int at = c + half;
          const float *src = !P.in_b ? P.in + row * P.cin + at
                                     : (at < P.planes_a ? P.in + row * P.planes_a + at : P.in_b + row * (P.cin - P.planes_a) + (at - P.planes_a));
          const float4 v = __ldg(reinterpret_cast<const float4 *>(src));
          x[half] = v.x, x[half + 1] = v.y, x[half + 2] = v.z, x[half + 3] = v.w;
          if (P.pre_scale) {
#pragma unroll
            for (int e = half; e < half + 4; ++e) {  // separate multiply and add, as the stand-alone BatchNorm kernel rounds them
              const float y = __fadd_rn(__fmul_rn(x[e], __ldg(P.pre_scale + c + e)), __ldg(P.pre_shift + c + e));
              x[e] = y * (y > 0.f ? 1.f : P.pre_leak);
            }
          }
        }
      split3_eight(x, P.rows + (row * (P.ppr * 8 / SP) + c / SP) * (size_t)(SP * 6) + c % SP * 2, SP * 2);
    } else {
      const int columns = P.cb * P.n_cb, n = (int)(idx % columns);
      const int c = (int)((idx / columns) % P.ppr) * 8, k = (int)(idx / ((long long)columns * P.ppr));
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (c + e < P.cin && n < P.cout) x[e] = __ldg(P.weight + ((long long)k * P.cin + c + e) * P.cout + n);
      const int nn = n % P.cb;
      const size_t part = (size_t)P.cb * SP * 2;
      split3_eight(x, P.image + (((size_t)k * P.n_cb + n / P.cb) * P.n_slices + c / SP) * 3 * part +
                          ((size_t)(nn / 8) * (SP / 8) + (c % SP) / 8) * 128 + (nn % 8) * 16, part);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) most = max(most, __float_as_uint(x[e]) & 0x7FFFFFFFu);
  }
  __shared__ unsigned all;
  if (threadIdx.x == 0) all = 0;
  __syncthreads();
  most = __reduce_max_sync(0xffffffffu, most);
  if ((threadIdx.x & 31) == 0) atomicMax(&all, most);
  __syncthreads();
  unsigned *range = rows ? P.in_range : P.w_range;
  for (int i = block + threadIdx.x * blocks; i < kRangeWords; i += kPrepareThreads * blocks) range[i] = all;
}

constexpr size_t kSmemBudget = 226 * 1024;

template <int SP, int NA>
int launch_six(SixParams &P, int n_sm, int dev, cudaStream_t stream) {
  static std::atomic<bool> configured[64];
  auto kernel = k_conv_six<SP, NA>;
  if (!configured[dev].load()) {
    SCN_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
    configured[dev].store(true);
  }
  const size_t stage = SixShape<SP>::A_BYTES + ((size_t)P.cb * SP * 6 + 1023) / 1024 * 1024;
  const size_t fixed = sizeof(int) * kSlots * kRows + kDrainWarps * kEpiBytes + sizeof(Ctl);
  P.n_stages = (int)std::min<size_t>(kMaxStages, (kSmemBudget - fixed) / stage);
  static_assert(SixWarps<NA>::THREADS >= kFmaGroups * kFmaGroup, "slow_items");
  SCN_REQUIRE((size_t)P.n_stages * stage + fixed - sizeof(Ctl) >= sizeof(float) * kFmaGroups * kFmaShare, SCN_ERR_UNSUPPORTED,
              "k_conv_six: %d stages of %zu bytes", P.n_stages, stage);
  P.per_tile = P.n_split * P.n_cb;
  P.n_items = P.n_tiles * P.per_tile;
  SCN_LAUNCH(kernel, (unsigned)std::min<long long>(P.n_items, (long long)n_sm), SixWarps<NA>::THREADS, kSmemBudget, stream, P);
  SCN_CUDA_CHECK(cudaGetLastError());
  return SCN_OK;
}

// Into how many parts a tile's offsets are divided: as in conv_tile.cu, the smallest estimate of (waves of items) x (steps of
// an item) in SM cycles, plus, with more than one part, the partial sums' traffic and the second launch.  The constants are empirical
// here too: against 1 to 16 parts on 36 layers of U-Nets within 5 % of the best on 32; 256 -> 128 planes on 57 k rows 266 us (one part:
// 234), 192 -> 96 on 18.6 k 103 (four: 94), 64 -> 32 on 40 k 41.5 (three: 38.8), 192 -> 224 strided 18.5 (four: 17.5).
int split_parts(long long n_tiles, int n_cb, int K, int n_slices, double step_cycles, int cout, int n_sm) {
  const double offsets = n_tiles >= 2 * n_sm ? 0.5 * K : 0.75 * K;
  double best = 0;
  int best_s = 1;
  for (int s = 1; s <= 16 && s <= K; ++s) {
    const double waves = (double)ceil_div(n_tiles * n_cb * s, n_sm);
    double t = waves * (offsets / s * n_slices * step_cycles + 2500.0);
    if (s > 1) t += 6000.0 + (s + 1.0) * n_tiles * kRows * cout * 4.0 / 3400.0;
    if (s == 1 || t < 0.95 * best) best = t, best_s = s;
  }
  return best_s;
}

}  // namespace

extern thread_local int g_drop_arrival;  // test hook (conv_tc.cu)

// Which fp32 convolutions run here instead of on k_conv_fma (which is left for few output planes on many rows, whose
// multiply-adds cost less than six bytes per input value and rule, and for little work, where its one launch is the shorter
// chain).  One layer, us of its launches on this kernel / on k_conv_fma.  27 offsets, submanifold, sphere shells; the error of each
// against float64 (2-norm, products of mixed sign):
//                 16->16     16->32     32->32     64->64     96->96     160->160       error (96->96)
//   600 rows      13.1/10.4  13.1/10.7  14.2/11.6  16.1/16.0  18.4/24.7  21.2/46.1      0.8e-7 / 2.0e-7
//   1 000         13.3/10.6  13.4/11.2  13.7/12.5  16.1/18.0  18.9/31.8  23.8/62.4      0.9e-7 / 2.6e-7
//   2 000         13.7/11.9  13.7/12.6  14.1/14.6  16.8/26.6  22.3/53.2  36.2/110       0.9e-7 / 3.4e-7
//   9 000         16.3/14.9  17.4/18.7  18.4/23.4  29.1/60.6  41.5/127   92.0/327       1.0e-7 / 3.5e-7
//   30 000        20.3/32.3  21.4/42.5  26.4/59.5  53.6/141   81.8/317   222/859        1.1e-7 / 5.3e-7
//   200 000       72/97      78/135     102/200    231/603    359/1 549  1 005/4 178    1.2e-7 / 5.4e-7
// Other filters:
//   3-D shapes, 99 000 rows, 27 offsets: 8->16 37/42, 16->16 37/51, 32->16 46/69, 16->32 40/64
//   2-D strokes, 92 000 rows, 9 offsets: 16->16 21/20, 32->16 25/27, 16->32 23/26, 24->32 27/32, 32->32 27/38
//   2-D, 25 offsets, 32 000 rows: 16->32 24/40, 32->32 30/57, 64->64 61/143; 4-D, 81 offsets, 60 000 rows: 32->32 72/226
//   3 / 2, 27 offsets, 48 000 rows: 16->32 27/42, 32->32 35/58, 64->64 69/152, 128->128 143/536
// Windows side by side (filter = stride), where a fine row has one rule (2 / 2; fine rows; a Convolution's coarse rows):
//   Deconvolution 32->16     32->32     48->32     64->32     64->48     96->48     64->64     96->96     128->128
//   4 000 rows                                                                      10.4/10.3  11.2/10.0  12.4/15.1
//   15 000                                                                          10.9/11.1  12.0/14.9  13.9/21.5
//   25 000        10.2/5.2   10.4/7.5   11.7/8.9   11.8/9.7   12.6/13.3  14.5/17.1  13.6/13.4
//   100 000       15.9/10.9  16.8/16.6  20.2/19.9  21.4/22.1  24.5/31.5  29.1/42.1  26.8/31.9
//   200 000       22.5/15.8  23.6/24.8  29.1/30.2  31.3/34.2  36.0/55.1  44.1/73.4  39.6/56.6
//   400 000                             53/59      56/69                            72/113     100/242    142/340
//   1 600 000     118/118    142/191    175/222    193/246    230/413    296/536    240/414
//   error         0.5/1.0e-7 0.5/1.0e-7 0.5/1.3e-7 0.5/1.4e-7 0.5/1.4e-7 0.6/1.8e-7 0.5/1.4e-7
//   Convolution   32->48     32->64     64->64     96->64     64->96     96->96     128->128
//   1 100 rows    12.2/9.6              14.5/9.4   15.8/14.4  15.4/10.9  16.9/14.8  17.1/20.0
//   5 400         12.7/18.3             16.6/23.0  19.3/31.9  17.5/24.7  20.9/33.0  25.6/66.2
//   21 000        16.8/23.1             22.3/30.6  28.5/40.0  24.3/48.2  31.0/68.6  38.7/92.7
//   55 000        26.6/38.7  28.7/40.3  50.7/63.7
//   109 000       48/53                 84/97      119/134    87/158     123/224    166/311
//   463 000       166/192    176/192    308/321
// (The lines are from a form of this kernel that took 10 to 40 % longer.  What comes here gains; some of what stays away would gain too:
// 8 -> 16 planes on 99 000 rows of shapes 11 %, 24 -> 32 with 9 offsets 17 %, Deconvolutions to 48 planes and more up to 45 %,
// Convolutions to 64 planes on more than 90 000 rows 4 to 13 %.)
// Its error is the smaller one, or the same, for every shape and table that comes here, 8 to 256 planes, products of mixed
// and of one sign, rows behind a ReLU (16->32 on 9 000 rows of one sign, where k_conv_fma's sums are in parts: 6.5e-8 and
// 6.1e-8, so not here).
bool conv_six_takes(const float *in, const float *in_b, int planes_a, const float *out, const float *bias, int K, int cin,
                    int cout, int groups, long long rows_in, long long rows_out, bool disjoint, bool transposed) {
  if (groups != 1 || K > kOrderMaxOffsets || cin % 4 != 0 || cout % 4 != 0 || cout > 256 || (in_b && planes_a % 4 != 0) ||
      ((uintptr_t)in | (uintptr_t)in_b | (uintptr_t)out | (uintptr_t)bias) % 16 != 0 || rows_in >= (1ll << 31) || rows_out >= (1ll << 31))
    return false;
  const double weights = (double)K * cin * cout;
  if (rows_out < 512 || (cin <= 16 && rows_out < 16384) || (cout <= 16 && rows_out > 131072) || weights < (K < 27 ? 9000 : 6900) ||
      weights * rows_out < (rows_out >= 2048 ? 80e6 : disjoint ? 220e6 : 160e6))
    return false;
  if (!disjoint) return true;
  if (!transposed) return cout > 64 || rows_out <= 90000;
  return cin * cout >= 20000 || (cin >= 96 && cin * cout >= 8000 && rows_out >= 40000);
}

// out [n_out, cout] = act((bias + sum_k in[table[k][.]] @ W[k]) * bn_scale + bn_shift) for the table that `ord` packs, the
// input optionally a join and behind a BatchNorm of its own.  The operands in parts take 6 bytes per value of rows and
// weights (0.6 GB for 64 planes on 1.6 M rows) that k_conv_fma does without: where they are not to be had, nothing has been
// launched and *no_memory is set.
int conv_forward_six(const float *in, long long n_in, float *out, long long n_out, const float *weight, const float *bias,
                     const float *bn_scale, const float *bn_shift, float leak, const RowOrder &ord, int K, int cin, int cout,
                     int *flags, cudaStream_t stream, const float *pre_scale, const float *pre_shift, float pre_leak,
                     const float *in_b, int planes_a, bool *no_memory) {
  if (n_out == 0) return SCN_OK;
  const int SP = (cin + 15) / 16 * 16 % 32 == 0 ? 32 : 16, n_slices = (cin + SP - 1) / SP, cinp = n_slices * SP;
  const int coutp = (cout + 15) / 16 * 16, n_cb = coutp > 128 ? 2 : 1, cb = n_cb == 1 ? coutp : (coutp / 2 + 15) / 16 * 16;
  int dev = 0;
  SCN_CUDA_CHECK(cudaGetDevice(&dev));
  SCN_REQUIRE(dev >= 0 && dev < 64, SCN_ERR_UNSUPPORTED, "device index %d unsupported", dev);
  static std::atomic<int> sm_count[64];
  int n_sm = sm_count[dev].load();
  if (!n_sm) {
    SCN_CUDA_CHECK(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    sm_count[dev].store(n_sm);
  }

  Scratch tmp(stream);
  unsigned char *image = nullptr, *rows = nullptr;
  const size_t image_bytes = (size_t)K * cinp * cb * n_cb * 6, rows_bytes = (size_t)std::max<long long>(n_in, 1) * cinp * 6;
  float *partial = nullptr;
  const double chunk = cb <= 64 ? std::max(56.0, 1.5 * cb) + std::max(56.0, 1.0 * cb) + 56 : 6 * std::max(56.0, 0.5 * cb);
  const double step = std::max((kRows * SP * 6.0 + cb * SP * 6.0) / 32.0, chunk * SP / 16);
  const char *e = getenv("SCN_SIX_SPLIT");
  const int n_split = e ? (int)std::max<long long>(1, std::min<long long>({atoi(e), 64, (1ll << 31) / (ord.n_tiles * kRows) - 1})) : split_parts(ord.n_tiles, n_cb, ord.one_offset ? 1 : K, n_slices, step, cout, n_sm);
  if (tmp.get(&image, image_bytes + sizeof(unsigned) * kRangeWords) != SCN_OK ||  // (multiples of 16)
      tmp.get(&rows, rows_bytes + sizeof(unsigned) * kRangeWords) != SCN_OK ||
      (n_split > 1 && tmp.get(&partial, (size_t)n_split * ord.n_tiles * kRows * cout * sizeof(float)) != SCN_OK)) {
    *no_memory = true;
    return SCN_OK;
  }
  PrepareParams Q{};
  Q.in = in;
  Q.in_b = in_b;
  Q.rows = rows;
  Q.in_range = (unsigned *)(rows + rows_bytes);
  Q.ppr = cinp / 8;
  Q.n_pieces = n_in * Q.ppr;
  Q.cin = cin;
  Q.planes_a = planes_a;
  Q.pre_scale = pre_scale;
  Q.pre_shift = pre_shift;
  Q.pre_leak = pre_leak;
  Q.weight = weight;
  Q.image = image;
  Q.w_range = (unsigned *)(image + image_bytes);
  Q.w_pieces = (long long)K * Q.ppr * cb * n_cb;
  Q.cout = cout;
  Q.cb = cb;
  Q.n_cb = n_cb;
  Q.n_slices = n_slices;
  Q.row_blocks = (int)std::max<long long>(1, std::min<long long>(ceil_div(Q.n_pieces, kPrepareThreads), kPrepareBlocks));
  const unsigned blocks = Q.row_blocks + (unsigned)std::min<long long>(ceil_div(Q.w_pieces, kPrepareThreads), kPrepareBlocks);
  const auto prepare = SP == 32 ? k_six_prepare<32> : k_six_prepare<16>;
  SCN_LAUNCH(prepare, blocks, kPrepareThreads, 0, stream, Q);

  SixParams P{};
  P.in_split = rows;
  P.in_range = Q.in_range;
  P.row_bytes = (long long)cinp * 6;
  P.n_in = n_in;
  P.out = out;
  P.cout = cout;
  P.cb = cb;
  P.n_cb = n_cb;
  P.wprep = image;
  P.w_range = Q.w_range;
  P.bias = bias;
  P.bn_scale = bn_scale;
  P.bn_shift = bn_shift;
  P.leak = bn_scale ? leak : 1.f;
  P.order = ord.order;
  P.packed = ord.packed;
  P.by_work = ord.by_work;
  P.tile_bits = ord.tile_bits;
  P.words = ord.words;
  P.K = K;
  P.n_slices = n_slices;
  P.log2_terms = bit_length((unsigned long long)K * cin);
  P.n_tiles = ord.n_tiles;
  P.in = in;
  P.in_b = in_b;
  P.weight = weight;
  P.pre_scale = pre_scale;
  P.pre_shift = pre_shift;
  P.pre_leak = pre_leak;
  P.cin = cin;
  P.planes_a = planes_a;
  P.flags = flags;
  P.drop = g_drop_arrival;
  g_drop_arrival = 0;
  P.n_split = n_split;
  if (n_split > 1) P.out = partial;
  const auto launch = SP == 32 ? (cb <= 32 ? launch_six<32, 16> : cb <= 64 ? launch_six<32, 32> : launch_six<32, 64>)
                               : (cb <= 32 ? launch_six<16, 16> : cb <= 64 ? launch_six<16, 32> : launch_six<16, 64>);
  SCN_TRY(launch(P, n_sm, dev, stream));
  if (n_split > 1)
    SCN_TRY(sum_partial_tiles(partial, n_split, P.n_tiles * kRows, cout, ord.order, n_out, bias, bn_scale, bn_shift, leak, out, stream));
  return SCN_OK;
}

}  // namespace scn
