// Sparse convolution on tcgen05 tensor cores over mask-sorted row tiles: the kernel of the bf16 modes (the
// fp32-class three-term form and the single-pass one).
//
// Same mathematics as the other convolution kernels (the reference's per-offset gather / GEMM / scatter-add is
// CPU/Convolution.cpp:137-148, CUDA/Convolution.cu:57-233): output stationary, each output row written once,
//     D[128 rows x planes] += G_k[128 rows x 32 planes] * W_k[32 planes x planes]
// with the gathered input rows as the MMA's A operand (M = 128 TMEM lanes = rows of the tile) and the weights as
// its B operand (N = output planes).
//
// What this form is built on:
//   * Tiles are packed from rows that have the same set of filter offsets (row_order.cu), so a tile of 128 rows
//     runs 9 to 12 steps of 27 instead of 22 to 25 and nearly every row of a step holds a rule.
//   * A tcgen05.mma takes max(56, N / 2) cycles for 128 rows (scn_tc_probe_mma) and reads both operands from shared memory.
//     With up to 128 output planes the slab [W_h | W_m] is one operand of 2 x planes columns: h (W_h | W_m) is ONE instruction
//     whose two column ranges are the large and one small term, m W_h goes to the small range, the epilogue adds the two:
//     2 instructions per 16 planes instead of 3, and the rows are read twice instead of three times.  (Above 64 planes too
//     since the reads count: U-Net on eight rooms 6095 -> 6034 us, on one room 1912 -> 1884.  The small terms are no longer cut
//     off against the large ones, so the error against float64 fell: 128 -> 128 planes on 60 k rows 6.6e-6 -> 4.7e-6, of one
//     sign 6.9e-6 -> 3.7e-6; smaller for every shape of 80 to 128 planes.)
//   * What bounds it is the gather: 128 bytes per row and 32-plane step (16 + 16 bits per value) through 16-byte
//     cp.async at about 32 bytes per cycle and SM, 512 cycles per step against 224 cycles of tensor work for 32
//     output planes, 304 for 96.
//
// Roles (15 warps, one CTA per SM, persistent).  A step is one filter offset of one tile and SP input planes; the
// steps of a CTA are numbered through all its tiles and step n uses stage n % n_stages of one ring.
//   entries     one thread: a slot per (tile, filter offset with a rule), the input row of every tile row, one 512-byte
//               bulk copy from the packed table; up to kSlots offsets ahead
//   producers   8 warps, warp w takes steps w, w + 8, ...: all 128 rows of the step by 16-byte cp.async pieces
//               straight into the swizzled operand layout, zero fill where a row has no rule; the barrier arrival
//               happens when a lane's copies have landed.  (One warp per step: with a step spread over all warps its
//               chain of waits and address arithmetic, longer than its copies take, was the time of the step: 1 500
//               cycles against the 512 the copies need.)
//   weights     one thread: one bulk copy per step
//   MMA         one thread
//   epilogue    4 warps: tcgen05.ld (a lane holds a row) -> shared memory, 16 planes at a time -> bias -> optional
//               BatchNorm scale / shift / leaky ReLU -> 16-byte stores, four lanes per row.  (Stored straight from the TMEM
//               lanes every instruction touched 32 lines: a fifth of the cycles in which the gather could have issued.)
//
// With fewer tiles than SMs the offsets of a tile are divided over n_split items whose partial sums are added in a
// fixed order (k_tile_sum).
//
// Every wait is bounded; on expiry the role raises the abort flag, everybody leaves, tensor memory is freed and
// the host sees FLAG_TC_TIMEOUT through scn_md_poll_errors.
#include <stdlib.h>

#include <algorithm>
#include <atomic>

#include "conv_tile.cuh"

namespace scn {

namespace {

constexpr int kRows = kOrderTile;  // rows of a tile = MMA M
constexpr int kProdWarps = 8;
constexpr int kEpi0 = kProdWarps, kMma = kProdWarps + 4, kWgt = kMma + 1, kEntries = kMma + 2;
constexpr int kThreads = (kProdWarps + 7) * 32;
constexpr int kSlots = 8;       // offsets the entries run ahead; at least kProdWarps (the slots that end the work)
constexpr int kMaxStages = 12;
constexpr int kEpiBytes = 32 * 64;  // per epilogue warp: 32 rows x 16 planes on their way from TMEM lanes to whole lines

struct TileParams {
  const unsigned char *in_split;  // split rows: per slice [SP h | SP m] (three-term) or [SP h]
  long long row_bytes;
  long long n_in;
  float *out;       // n_split == 1: [n_out][cout]; else partial sums [n_split][n_tiles * 128][cout]
  long long n_out;
  int cout, coutp;  // coutp: output planes rounded up to 16 (the operand image's)
  const unsigned char *wprep;
  const float *bias, *bn_scale, *bn_shift;
  float leak;
  const int *order, *packed, *by_work;
  const unsigned *tile_bits;
  int words;
  int K, n_slices;
  int n_stages, tmem_cols;
  long long n_tiles, n_items;
  int n_split;
  unsigned char *out_split;  // (optional, n_split 1) the result once more as split rows, slices of out_sp planes
  int out_sp;
  int drop;         // test hook: leave out one barrier arrival of the first CTA
  int *flags;
};

template <int TERMS, int SP>
struct TileShape {
  static constexpr int PARTS = TERMS == 3 ? 2 : 1;
  static constexpr int PP = SP * 2 * PARTS / 16;      // 16-byte pieces per row and step
  static constexpr int NI = kRows / (32 / PP);        // copy instructions per step and lane
  static constexpr unsigned ROW = PP * 16;            // bytes of a row in a stage: 128 or 64
  static constexpr unsigned A_BYTES = kRows * ROW;
  static_assert(PP == 8 || PP == 4, "a row of a step is 128 or 64 bytes");
};

// control block behind the ring
struct Ctl {
  unsigned long long full[kMaxStages], empty[kMaxStages];  // rows and weights landed; MMAs done
  unsigned long long s_full[kSlots], s_empty[kSlots], acc_full[4], acc_empty[4];
  int slot_k[kSlots];  // filter offset of the slot; -1: no more work; kNoRules: offset 0 with rows of zeros
  unsigned tmem;
  int abort;
};

// The tile of an item: the tiles with the most offsets first (packed tiles come in ascending order of their masks, so from
// the back where they have not been sorted by work).
__device__ __forceinline__ long long item_tile(const TileParams &P, long long item) {
  const long long i = P.n_split == 1 ? item : item / P.n_split;
  return P.by_work ? __ldg(P.by_work + i) : P.n_tiles - 1 - i;
}

// filter offsets of an item: those of its tile, or its share of them when the offsets are divided
__device__ __forceinline__ int item_offsets(const TileParams &P, long long item) {
  if (item >= P.n_items) return 0;
  const long long t = item_tile(P, item);
  int total = 0;
  for (int w = 0; w < P.words; ++w) total += __popc(__ldg(P.tile_bits + t * P.words + w));
  if (P.n_split == 1) return total;
  const int part = (int)(item % P.n_split);
  return total * (part + 1) / P.n_split - total * part / P.n_split;
}

template <int TERMS, int SP, bool OUT_SPLIT>
__global__ void __launch_bounds__(kThreads, 2) k_conv_tile(TileParams P) {
  SCN_GRID_WAIT();
  using Shape = TileShape<TERMS, SP>;
  constexpr int PP = Shape::PP, NI = Shape::NI, PARTS = Shape::PARTS;
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned w_part = (unsigned)P.coutp * SP * 2;  // one bf16 weight slab
  const unsigned w_bytes = w_part * PARTS;
  const unsigned stage_bytes = Shape::A_BYTES + ((w_bytes + 1023u) & ~1023u);  // the swizzle pattern repeats every 1 KB
  const unsigned smem0 = smem_u32(smem);
  unsigned char *tail = smem + (size_t)P.n_stages * stage_bytes;
  int *entries = reinterpret_cast<int *>(tail);  // [kSlots][128] input row of every tile row, or -1
  unsigned char *epi = tail + sizeof(int) * kSlots * kRows;
  Ctl &C = *reinterpret_cast<Ctl *>(epi + 4 * kEpiBytes);
  const bool joint = TERMS == 3 && P.coutp <= 128;  // [W_h | W_m] as one operand
  const int dcols = ((joint ? 2 : 1) * P.coutp + 31) & ~31;
  const int n_acc = min(4, P.tmem_cols / dcols);

  if (tid == 0) {
    for (int i = 0; i < P.n_stages; ++i) {
      mbar_init(&C.full[i], 32 + 1);  // the producing warp's lanes and the weights
      mbar_init(&C.empty[i], 1);
    }
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&C.s_full[i], 1);
      mbar_init(&C.s_empty[i], P.n_slices + 1);    // a producer warp per slice, and the weights
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&C.acc_full[i], 1);
      mbar_init(&C.acc_empty[i], 4);
    }
    C.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMma) tmem_alloc(&C.tmem, (unsigned)P.tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = C.tmem;
  volatile int *abort = &C.abort;
  const long long my_items = items_here(P.n_items);  // (the grid has at most n_items CTAs)

  if (warp < kProdWarps) {
    // ==================================== producers =============================================
    // this lane's 16-byte piece of the rows q NI .. q NI + NI - 1 (the entries of a lane follow one another)
    const int j = lane % PP, q = lane / PP;
    const unsigned lane_dst = (unsigned)(q * NI) * Shape::ROW + (unsigned)j * 16;
    // No more warps than stages: a warp at step n has seen the consumption of step n - active - n_stages, and its wait
    // below can tell step n - n_stages from the one a round earlier only if that one is not later than this.
    const int active = min(kProdWarps, P.n_stages);
    const int d_slot = active / P.n_slices, d_slice = active % P.n_slices;
    const int d_round = active / P.n_stages, d_st = active % P.n_stages;
    int slot = warp / P.n_slices, slice = warp % P.n_slices;
    int round = warp / P.n_stages, st = warp % P.n_stages;
    bool ok = true, bad = false;
    while (warp < active) {
      const int si = slot % kSlots;
      if (!mbar_wait(&C.s_full[si], (slot / kSlots) & 1)) {
        ok = false;
        break;
      }
      const int slot_k = C.slot_k[si];
      if (slot_k < 0 || *abort) break;
      const int rows_in = slot_k == kNoRules ? 0 : (int)P.n_in;  // entries below it are rows
      const int4 *ent = reinterpret_cast<const int4 *>(entries + si * kRows + q * NI);
      if (!mbar_wait(&C.empty[st], (round + 1) & 1)) {  // (the first round passes)
        ok = false;
        break;
      }
      const unsigned dst = smem0 + (unsigned)st * stage_bytes + lane_dst;
      const unsigned char *col = P.in_split + slice * (SP * 2 * PARTS) + j * 16;
#pragma unroll
      for (int i = 0; i < NI; i += 4) {
        const int4 e4 = ent[i / 4];
        const int v[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const bool hit = (unsigned)v[e] < (unsigned)rows_in;
          bad |= v[e] >= (int)P.n_in && slot_k != kNoRules;
          const unsigned swizzle = (PP == 8 ? (i + e) & 7 : ((i + e) >> 1) & 3) * 16;  // (q NI is a multiple of eight)
          cp_async16((dst ^ swizzle) + (i + e) * Shape::ROW, col + (size_t)(unsigned)(hit ? v[e] : 0) * P.row_bytes, hit ? 16u : 0u);
        }
      }
      cp_async_arrive(&C.full[st]);
      __syncwarp();
      if (lane == 0) mbar_arrive(&C.s_empty[si]);
      slot += d_slot, slice += d_slice;
      if (slice >= P.n_slices) slice -= P.n_slices, ++slot;
      round += d_round, st += d_st;
      if (st >= P.n_stages) st -= P.n_stages, ++round;
    }
    if (bad) atomicOr(P.flags, FLAG_BAD_ROW);
    asm volatile("cp.async.wait_all;" ::: "memory");  // they must land before the CTA's shared memory goes away
    if (!ok) *abort = 1;
  } else if (warp == kWgt) {
    // ==================================== weights ===============================================
    if (lane == 0) {
      int st = 0, par = 1;
      long long filled = 0;
      bool ok = true;
      for (int slot = 0; ok; ++slot) {
        const int si = slot % kSlots;
        if (!mbar_wait(&C.s_full[si], (slot / kSlots) & 1)) {
          ok = false;
          break;
        }
        const int k = C.slot_k[si];
        mbar_arrive(&C.s_empty[si]);
        if (k < 0) break;
        const unsigned char *src = P.wprep + (size_t)(k == kNoRules ? 0 : k) * P.n_slices * w_bytes;
        for (int s = 0; s < P.n_slices; ++s) {
          if (!mbar_wait(&C.empty[st], par) || *abort) {
            ok = false;
            break;
          }
          if (!(P.drop && blockIdx.x == 0 && filled == 0)) {
            mbar_expect_tx(&C.full[st], w_bytes);
            bulk_copy_g2s(smem0 + (unsigned)st * stage_bytes + Shape::A_BYTES, src + (size_t)s * w_bytes, w_bytes, &C.full[st]);
          }
          ++filled;
          if (++st == P.n_stages) st = 0, par ^= 1;
        }
      }
      if (!ok) {  // slabs in flight must land before the CTA's shared memory goes away
        *abort = 1;
        for (int i = 0; i < P.n_stages; ++i) {
          const long long uses = (filled + P.n_stages - 1 - i) / P.n_stages;
          if (uses > 0) mbar_wait(&C.full[i], (unsigned)((uses - 1) & 1));
        }
      }
    }
  } else if (warp == kMma) {
    // ==================================== MMA issue =============================================
    // The whole warp runs the loop and one elected lane issues: with warp-uniform control flow and operands (votes and
    // reductions instead of loaded flags) the descriptors stay in uniform registers.  Issued from inside a lane == 0
    // branch every instruction cost 200 to 260 cycles of moves and address arithmetic, four to eight times its own.
    const unsigned id_all = tile_idesc(joint ? 2 * P.coutp : P.coutp), id_one = tile_idesc(P.coutp);
    const unsigned long long a_desc = rows_desc<Shape::ROW>(smem0, 0);
    const unsigned long long w_desc = smem_desc(smem0 + Shape::A_BYTES, 128, SP / 8 * 128);
    const unsigned a_hi = (unsigned)(a_desc >> 32), w_hi = (unsigned)(w_desc >> 32);
    const unsigned a0 = (unsigned)a_desc, w0 = (unsigned)w_desc;
    const unsigned stage_step = stage_bytes >> 4, wm_step = w_part >> 4;
    const int items = (int)my_items, n_stages = P.n_stages, coutp = P.coutp;
    int st = 0, par = 0, buf = 0, buf_par = 1;
    unsigned at = 0, d = tmem;
    bool ok = true;
    const bool leader = elect_one();
    int offsets_next = item_offsets(P, item_of(0));
    for (int i = 0; i < items && ok; ++i) {
      const int steps = __reduce_max_sync(0xffffffffu, max(1, offsets_next)) * P.n_slices;
      offsets_next = item_offsets(P, item_of(i + 1));
      // the item's accumulator must have been drained
      if (!mbar_wait_warp(&C.acc_empty[buf], buf_par) || __any_sync(0xffffffffu, *abort != 0)) {
        ok = false;
        break;
      }
      for (int s = 0; s < steps; ++s) {
        if (!mbar_wait_warp(&C.full[st], par)) {
          ok = false;
          break;
        }
        if (leader) {
          // order the copied rows (acquired through the barrier) before the tensor core's async-proxy reads; done
          // here, not by the producers: their fence would wait for the copies they have just started
          fence_proxy_async_smem();
          tc_fence_after();
#pragma unroll
          for (int jj = 0; jj < SP / 16; ++jj) {
            const unsigned ah = a0 + at + jj * 2, am = ah + SP / 8, wh = w0 + at + jj * 16;
            if (jj == 0) mma_bf16(d, ah, a_hi, wh, w_hi, joint ? id_all : id_one, (unsigned)s);
            else mma_bf16_acc(d, ah, a_hi, wh, w_hi, joint ? id_all : id_one);
            if (TERMS == 3) {
              if (joint) {
                mma_bf16_acc(d + coutp, am, a_hi, wh, w_hi, id_one);
              } else {
                mma_bf16_acc(d, ah, a_hi, wh + wm_step, w_hi, id_one);
                mma_bf16_acc(d, am, a_hi, wh, w_hi, id_one);
              }
            }
          }
          tc_commit(&C.empty[st]);
          if (s == steps - 1) tc_commit(&C.acc_full[buf]);
        }
        __syncwarp();
        at += stage_step;
        if (++st == n_stages) st = 0, par ^= 1, at = 0;
      }
      d += dcols;
      if (++buf == n_acc) buf = 0, buf_par ^= 1, d = tmem;
    }
    if (!ok) *abort = 1;
  } else if (warp == kEntries) {
    // ==================================== entries ===============================================
    if (lane == 0) {
      int slot = 0;
      bool ok = true;
      unsigned b_next[4];
      auto fetch = [&](long long item) {
#pragma unroll
        for (int w = 0; w < 4; ++w)
          b_next[w] = item < P.n_items && w < P.words ? __ldg(P.tile_bits + item_tile(P, item) * P.words + w) : 0u;
      };
      fetch(item_of(0));
      for (long long it = 0; it < my_items && ok; ++it) {
        const long long item = item_of(it);
        unsigned u[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) u[w] = b_next[w];
        fetch(item_of(it + 1));
        const int *src = P.packed + item_tile(P, item) * P.K * kRows;
        if (P.n_split > 1) {
          const int total = __popc(u[0]) + __popc(u[1]) + __popc(u[2]) + __popc(u[3]), part = (int)(item % P.n_split);
          const int first = total * part / P.n_split;
          keep_range(u, first, total * (part + 1) / P.n_split);
          src += first * kRows;
        }
        // a tile (or part) without any rule still gets one step, of weights and rows of zeros
        bool none = (u[0] | u[1] | u[2] | u[3]) == 0;
        if (none) u[0] = 1u;
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
            C.slot_k[si] = none ? kNoRules : w * 32 + __ffs(m) - 1;
            if (none) {
              mbar_arrive(&C.s_full[si]);
            } else {
              mbar_expect_tx(&C.s_full[si], kRows * 4);
              bulk_copy_g2s(smem_u32(entries + si * kRows), src, kRows * 4, &C.s_full[si]);
            }
          }
        }
      }
      const int filled = slot;
      // every producer warp finds its next step in a slot that ends it
      const int ends = (min(kProdWarps, P.n_stages) - 1) / P.n_slices + 1;
      for (int i = 0; i < ends && ok; ++i, ++slot) {
        const int si = slot % kSlots;
        if (!mbar_wait(&C.s_empty[si], ((slot / kSlots) + 1) & 1)) {
          ok = false;
          break;
        }
        C.slot_k[si] = -1;
        mbar_arrive(&C.s_full[si]);
      }
      if (!ok) {  // copies in flight must land before the CTA's shared memory goes away
        *abort = 1;
        for (int i = 0; i < kSlots; ++i) {
          const int uses = (filled + kSlots - 1 - i) / kSlots;
          if (uses > 0) mbar_wait(&C.s_full[i], (unsigned)((uses - 1) & 1));
        }
      }
    }
  } else {
    // ==================================== epilogue ==============================================
    const int quad = warp & 3;
    const int nc = P.cout;
    float4 *my_epi = reinterpret_cast<float4 *>(epi + quad * kEpiBytes);
    int buf = 0, buf_par = 0;
    for (long long it = 0; it < my_items; ++it) {
      const long long item = item_of(it), t = item_tile(P, item);
      const int part = (int)(item % P.n_split);
      const int orow = __ldg(P.order + t * kRows + quad * 32 + lane);
      int got = 1;
      if (lane == 0) got = (!*abort && mbar_wait(&C.acc_full[buf], buf_par)) ? 1 : 0;
      got = __shfl_sync(0xffffffffu, got, 0);
      if (!got) {
        *abort = 1;
        break;
      }
      tc_fence_after();
      const unsigned base = tmem + ((unsigned)(quad * 32) << 16) + (unsigned)(buf * dcols);
      // where rows lane / 4, + 8, + 16, + 24 of the warp go: this lane's four planes of them, or (OUT_SPLIT, which is short of
      // registers) the row.  Two CTAs of 15 warps have 64 registers a thread, and which form fits them was measured: 32 planes
      // on 200 k rows 51 us in both kernels, 56 with rows and eight columns at a time where nothing is split; 160 planes on
      // 3 k rows 24 us, 26 with rows and sixteen columns.
      long long at[4];
      int to[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = __shfl_sync(0xffffffffu, orow, i * 8 + (lane >> 2));
        if (OUT_SPLIT) to[i] = r;
        else at[i] = r < 0 ? -1 : (P.n_split > 1 ? ((long long)part * P.n_tiles + t) * kRows + quad * 32 + i * 8 + (lane >> 2) : r) * nc + (lane & 3) * 4;
      }
      for (int c0 = 0; c0 < nc; c0 += 16) {
        constexpr int kCols = OUT_SPLIT ? 8 : 16;
#pragma unroll
        for (int half = 0; half < 16; half += kCols) {
          unsigned a[kCols], b[kCols];
          if constexpr (OUT_SPLIT) {
            tmem_ld8_nowait(base + c0 + half, a);
            if (joint) tmem_ld8_nowait(base + P.coutp + c0 + half, b);
          } else {
            tmem_ld16_nowait(base + c0, a);
            if (joint) tmem_ld16_nowait(base + P.coutp + c0, b);
          }
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < kCols; e += 4) {
            float4 v;
            v.x = __uint_as_float(a[e]), v.y = __uint_as_float(a[e + 1]), v.z = __uint_as_float(a[e + 2]), v.w = __uint_as_float(a[e + 3]);
            if (joint) {
              v.x += __uint_as_float(b[e]), v.y += __uint_as_float(b[e + 1]);
              v.z += __uint_as_float(b[e + 2]), v.w += __uint_as_float(b[e + 3]);
            }
            my_epi[lane * 4 + (((half + e) >> 2) ^ ((lane >> 1) & 3))] = v;
          }
        }
        __syncwarp();
        const int c = c0 + (lane & 3) * 4;
        if (c < nc) {
          float4 bias = make_float4(0.f, 0.f, 0.f, 0.f), sc = bias, sh = bias;
          const bool finish = OUT_SPLIT || P.n_split == 1;
          if (finish && P.bias) bias = __ldg(reinterpret_cast<const float4 *>(P.bias + c));
          if (finish && P.bn_scale) {
            sc = __ldg(reinterpret_cast<const float4 *>(P.bn_scale + c));
            sh = __ldg(reinterpret_cast<const float4 *>(P.bn_shift + c));
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int row = i * 8 + (lane >> 2);
            float4 v = my_epi[row * 4 + ((lane & 3) ^ ((row >> 1) & 3))];
            if (OUT_SPLIT ? to[i] < 0 : at[i] < 0) continue;
            if (finish && P.bias) v.x += bias.x, v.y += bias.y, v.z += bias.z, v.w += bias.w;
            if (finish && P.bn_scale) {  // separate multiply and add, as the stand-alone BatchNorm kernel rounds them
              v.x = __fadd_rn(__fmul_rn(v.x, sc.x), sh.x), v.y = __fadd_rn(__fmul_rn(v.y, sc.y), sh.y);
              v.z = __fadd_rn(__fmul_rn(v.z, sc.z), sh.z), v.w = __fadd_rn(__fmul_rn(v.w, sc.w), sh.w);
              v.x *= v.x > 0.f ? 1.f : P.leak, v.y *= v.y > 0.f ? 1.f : P.leak;
              v.z *= v.z > 0.f ? 1.f : P.leak, v.w *= v.w > 0.f ? 1.f : P.leak;
            }
            *reinterpret_cast<float4 *>(P.out + (OUT_SPLIT ? (long long)to[i] * nc + c : at[i] + c0)) = v;
            if (OUT_SPLIT) {
              uint2 h, m;
              split_bf16_pair(v.x, v.y, h.x, m.x);
              split_bf16_pair(v.z, v.w, h.y, m.y);
              const int slice = c0 & -P.out_sp;  // (16, 32 or 64 planes)
              unsigned char *q = P.out_split + ((long long)to[i] * nc + slice) * (2 * PARTS) + (c - slice) * 2;
              *reinterpret_cast<uint2 *>(q) = h;
              if (PARTS == 2) *reinterpret_cast<uint2 *>(q + P.out_sp * 2) = m;
            }
          }
        }
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&C.acc_empty[buf]);
      if (++buf == n_acc) buf = 0, buf_par ^= 1;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort && tid == 0) atomicOr(P.flags, FLAG_TC_TIMEOUT);
  if (warp == kMma) tmem_dealloc(tmem, (unsigned)P.tmem_cols);
}

// partial [n_split][n_tiles * 128][cout] -> out: the parts of a row added in order, then bias and BatchNorm
__global__ void __launch_bounds__(256)
k_tile_sum(const float4 *__restrict__ partial, int n_split, long long n_pos, int cout4, const int *__restrict__ order,
           long long n_out, const float *__restrict__ bias, const float *__restrict__ bn_scale, const float *__restrict__ bn_shift,
           float leak, float4 *__restrict__ out, unsigned char *__restrict__ out_split, int out_sp, int parts) {
  SCN_GRID_WAIT();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_pos * cout4) return;
  const int c = (int)(i % cout4);
  const long long r = order ? __ldg(order + i / cout4) : i / cout4;
  if (r < 0 || r >= n_out) return;
  float4 q = __ldg(partial + i);
  for (int p = 1; p < n_split; ++p) {
    const float4 a = __ldg(partial + (long long)p * n_pos * cout4 + i);
    q.x += a.x, q.y += a.y, q.z += a.z, q.w += a.w;
  }
  if (bias) {
    const float4 b4 = __ldg(reinterpret_cast<const float4 *>(bias) + c);
    q.x += b4.x, q.y += b4.y, q.z += b4.z, q.w += b4.w;
  }
  if (bn_scale) {
    const float4 sc = __ldg(reinterpret_cast<const float4 *>(bn_scale) + c), sh = __ldg(reinterpret_cast<const float4 *>(bn_shift) + c);
    q.x = __fadd_rn(__fmul_rn(q.x, sc.x), sh.x), q.y = __fadd_rn(__fmul_rn(q.y, sc.y), sh.y);
    q.z = __fadd_rn(__fmul_rn(q.z, sc.z), sh.z), q.w = __fadd_rn(__fmul_rn(q.w, sc.w), sh.w);
    q.x *= q.x > 0.f ? 1.f : leak, q.y *= q.y > 0.f ? 1.f : leak;
    q.z *= q.z > 0.f ? 1.f : leak, q.w *= q.w > 0.f ? 1.f : leak;
  }
  out[r * cout4 + c] = q;
  if (out_split) {
    uint2 h, m;
    split_bf16_pair(q.x, q.y, h.x, m.x);
    split_bf16_pair(q.z, q.w, h.y, m.y);
    unsigned char *s = out_split + (r * cout4 * 4 + c * 4 / out_sp * out_sp) * (2 * parts) + c * 4 % out_sp * 2;
    *reinterpret_cast<uint2 *>(s) = h;
    if (parts == 2) *reinterpret_cast<uint2 *>(s + out_sp * 2) = m;
  }
}

// in [n][cin] fp32 (or the column-wise concatenation [in (planes_a) | in_b], read where the two lie) -> per row and
// slice of SP planes [SP h | SP m], h = bf16(x), m = bf16(x - h); PARTS 1: only h.  Planes past cin are zero.  One
// thread per 8 planes.  pre_scale / pre_shift: x first goes through an eval-mode BatchNorm and its leaky ReLU, with
// the roundings of the stand-alone operator.  Bound by HBM: 32 bytes in, 16 x PARTS out per thread.
template <int PARTS>
__global__ void __launch_bounds__(256)
k_tile_split(const float *__restrict__ in, unsigned char *__restrict__ out, long long n_pieces, int cin, int ppr, int SP,
             const float *__restrict__ pre_scale, const float *__restrict__ pre_shift, float pre_leak,
             const float *__restrict__ in_b, int planes_a) {
  SCN_GRID_WAIT();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n_pieces) return;
  const long long row = idx / ppr;
  const int piece = (int)(idx - row * ppr), c = piece * 8, slice = c / SP, j = (c % SP) / 8;
  float x[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) x[e] = 0.f;
  if (c < cin) {
    const float *src = !in_b ? in + row * cin + c
                             : (c < planes_a ? in + row * planes_a + c : in_b + row * (cin - planes_a) + (c - planes_a));
    const float4 a = __ldg(reinterpret_cast<const float4 *>(src)), b = __ldg(reinterpret_cast<const float4 *>(src) + 1);
    x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w, x[4] = b.x, x[5] = b.y, x[6] = b.z, x[7] = b.w;
    if (pre_scale) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float y = __fadd_rn(__fmul_rn(x[e], __ldg(pre_scale + c + e)), __ldg(pre_shift + c + e));
        x[e] = y * (y > 0.f ? 1.f : pre_leak);
      }
    }
  }
  uint4 h, m;
  split_bf16_pair(x[0], x[1], h.x, m.x);
  split_bf16_pair(x[2], x[3], h.y, m.y);
  split_bf16_pair(x[4], x[5], h.z, m.z);
  split_bf16_pair(x[6], x[7], h.w, m.w);
  unsigned char *q = out + (row * (ppr * 8 / SP) + slice) * (size_t)(SP * 2 * PARTS) + j * 16;
  *reinterpret_cast<uint4 *>(q) = h;
  if (PARTS == 2) *reinterpret_cast<uint4 *>(q + SP * 2) = m;
}

// W [K][cin][cout] -> [K][slice][part][coutp x SP] bf16 in the K-major core-matrix layout of the MMA's B operand
__global__ void k_tile_weights(const float *__restrict__ w, unsigned char *__restrict__ out, int K, int cin, int cout,
                               int coutp, int n_slices, int SP, int parts) {
  SCN_GRID_WAIT();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int cp = n_slices * SP;
  if (idx >= (long long)K * cp * coutp) return;
  const int n = (int)(idx % coutp), c = (int)((idx / coutp) % cp), k = (int)(idx / ((long long)coutp * cp));
  const float v = (c < cin && n < cout) ? w[((long long)k * cin + c) * cout + n] : 0.f;
  const int slice = c / SP, kk = c % SP;
  const size_t tile = (size_t)coutp * SP * 2;
  const size_t off = (size_t)(n / 8) * (SP / 8) * 128 + (size_t)(kk / 8) * 128 + (n % 8) * 16 + (kk % 8) * 2;
  unsigned char *base = out + ((size_t)k * n_slices + slice) * parts * tile;
  const __nv_bfloat16 h = __float2bfloat16_rn(v);
  *reinterpret_cast<__nv_bfloat16 *>(base + off) = h;
  if (parts == 2) *reinterpret_cast<__nv_bfloat16 *>(base + tile + off) = __float2bfloat16_rn(v - __bfloat162float(h));
}

constexpr size_t kSmemBudget = 226 * 1024;

// planes per step: as wide as the row allows (fewer steps, longer contiguous reads) without padding it further than
// to a multiple of 16 (32 with single parts)
int slice_planes(int terms, int cin) {
  const int c = (cin + 15) / 16 * 16;
  if (terms == 1) return c % 64 == 0 ? 64 : 32;
  return c % 32 == 0 ? 32 : 16;
}

template <int TERMS, int SP, bool OUT_SPLIT>
int launch_tile_as(TileParams &P, int n_sm, int dev, cudaStream_t stream) {
  using Shape = TileShape<TERMS, SP>;
  static std::atomic<bool> configured[64];
  auto kernel = k_conv_tile<TERMS, SP, OUT_SPLIT>;
  if (!configured[dev].load()) {
    SCN_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
    configured[dev].store(true);
  }
  const size_t stage = Shape::A_BYTES + ((size_t)P.coutp * SP * 2 * Shape::PARTS + 1023) / 1024 * 1024;
  const size_t fixed = sizeof(int) * kSlots * kRows + 4 * kEpiBytes + sizeof(Ctl);
  const int dcols = ((TERMS == 3 && P.coutp <= 128 ? 2 : 1) * P.coutp + 31) & ~31;
  // Two CTAs per SM, each with half of the shared memory and of the TMEM columns, where that leaves four stages and two
  // accumulators: one CTA's issue overhead and epilogue run beside the other's tensor instructions.
  int ctas = dcols * 2 <= 256 && (kSmemBudget / 2 - fixed) / stage >= 4 ? 2 : 1;
  if (const char *e = getenv("SCN_TILE_CTAS")) ctas = atoi(e) == 2 && dcols <= 256 && (kSmemBudget / 2 - fixed) / stage >= 2 ? 2 : 1;
  const size_t smem = kSmemBudget / ctas / 1024 * 1024;
  P.tmem_cols = 512 / ctas;
  P.n_stages = (int)std::min<size_t>(kMaxStages, (smem - fixed) / stage);
  SCN_REQUIRE(P.n_stages >= 2, SCN_ERR_UNSUPPORTED, "tile kernel: %d output planes do not fit shared memory", P.cout);
  P.n_items = P.n_tiles * P.n_split;
  SCN_LAUNCH(kernel, (unsigned)std::min<long long>(P.n_items, (long long)n_sm * ctas), kThreads, smem, stream, P);
  SCN_CUDA_CHECK(cudaGetLastError());
  return SCN_OK;
}

template <int TERMS, int SP>
int launch_tile(TileParams &P, int n_sm, int dev, cudaStream_t stream) {
  return P.out_split ? launch_tile_as<TERMS, SP, true>(P, n_sm, dev, stream) : launch_tile_as<TERMS, SP, false>(P, n_sm, dev, stream);
}

}  // namespace

// out = act((bias + the parts of partial [n_split][n_pos][cout], in order) * bn_scale + bn_shift); position p is row
// order[p] (order null: row p).  out_split (optional): the result as split rows as well, see k_tile_split
int sum_partial_tiles(const float *partial, int n_split, long long n_pos, int cout, const int *order, long long n_out,
                      const float *bias, const float *bn_scale, const float *bn_shift, float leak, float *out,
                      cudaStream_t stream, unsigned char *out_split, int out_sp, int parts) {
  SCN_LAUNCH(k_tile_sum, (unsigned)ceil_div(n_pos * (cout / 4), 256), 256, 0, stream, (const float4 *)partial, n_split, n_pos, cout / 4, order, n_out, bias, bn_scale, bn_shift, leak, (float4 *)out, out_split, out_sp, parts);
  SCN_CUDA_CHECK(cudaGetLastError());
  return SCN_OK;
}

extern thread_local int g_drop_arrival;  // test hook (conv_tc.cu)

bool conv_tile_supported(const float *in, const float *in_b, int planes_a, const float *out, const float *bias, int K,
                         int cin, int cout, int groups) {
  return groups == 1 && K <= kOrderMaxOffsets && cin % 8 == 0 && cin >= 8 && cout % 8 == 0 && cout >= 8 && cout <= 256 &&
         (!in_b || planes_a % 8 == 0) && ((uintptr_t)in | (uintptr_t)in_b | (uintptr_t)out | (uintptr_t)bias) % 16 == 0;
}

// Into how many parts a tile's offsets are divided: the smallest estimate of (waves of items) x (steps of an item),
// plus, with more than one part, the partial sums' traffic and the second launch.  In SM cycles; a step is bound by its
// 16 KB of gathered rows at 32 bytes per cycle or by its weight slab, an item also costs the fill and drain of the rings.
static int split_parts(long long n_tiles, int K, int n_slices, double step_cycles, int cout, int n_sm) {
  const double offsets = n_tiles >= 2 * n_sm ? 0.5 * K : 0.75 * K;  // sorted tiles of a large level meet fewer
  double best = 0;
  int best_s = 1;
  for (int s = 1; s <= 16 && s <= K; ++s) {
    const double waves = (double)ceil_div(n_tiles * s, n_sm);
    double t = waves * (offsets / s * n_slices * step_cycles + 2500.0);
    if (s > 1) t += 6000.0 + (s + 1.0) * n_tiles * kRows * cout * 4.0 / 3400.0;
    if (s == 1 || t < 0.95 * best) best = t, best_s = s;
  }
  return best_s;
}

// out [n_out, cout] = act((bias + sum_k in[table[k][.]] @ W[k]) * bn_scale + bn_shift) for the table that `ord` packs, the
// input optionally a join and behind a BatchNorm of its own (see k_tile_split)
int conv_forward_tile(const float *in, long long n_in, float *out, long long n_out, const float *weight,
                      const float *bias, const float *bn_scale, const float *bn_shift, float leak,
                      const RowOrder &ord, int K, int cin, int cout, int precision, int *flags, cudaStream_t stream,
                      const float *pre_scale, const float *pre_shift, float pre_leak, const float *in_b, int planes_a) {
  if (n_out == 0) return SCN_OK;
  SCN_REQUIRE(n_in < (1ll << 31) && n_out < (1ll << 31), SCN_ERR_UNSUPPORTED, "row count above 2^31");
  const int terms = precision == SCN_PRECISION_BF16 ? 1 : 3, parts = terms == 3 ? 2 : 1;
  const int SP = slice_planes(terms, cin), n_slices = (cin + SP - 1) / SP, cinp = n_slices * SP;
  const int coutp = (cout + 15) / 16 * 16;
  int dev = 0;
  SCN_CUDA_CHECK(cudaGetDevice(&dev));
  SCN_REQUIRE(dev >= 0 && dev < 64, SCN_ERR_UNSUPPORTED, "device index %d unsupported", dev);
  static std::atomic<int> sm_count[64];
  int n_sm = sm_count[dev].load();
  if (!n_sm) {
    SCN_CUDA_CHECK(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    sm_count[dev].store(n_sm);
  }

  struct Image : WeightImage {
    cudaStream_t stream;
    ~Image() { weight_image_put(*this, stream); }
  } wi;
  wi.stream = stream;
  bool build = true;
  SCN_TRY(weight_image_get(WIMG_TILE, K, cin, cout, SP * 4 + parts, (size_t)K * cinp * coutp * 2 * parts, stream, &wi, &build));
  if (build)
    SCN_LAUNCH(k_tile_weights, (unsigned)ceil_div((long long)K * cinp * coutp, 256), 256, 0, stream, weight,
               (unsigned char *)wi.ptr, K, cin, cout, coutp, n_slices, SP, parts);

  // the input rows as bf16 parts, made once per call: a row is gathered by up to K output rows.  The layer that made the
  // rows may have left them in this form already, and the next one may want them so.
  const SplitRows rows = take_split_rows();
  Scratch tmp(stream);
  unsigned char *split = nullptr;
  const bool given = rows.in && !pre_scale && !in_b && cinp == cin;
  if (!given) SCN_TRY(tmp.get(&split, (size_t)std::max<long long>(n_in, 1) * cinp * 2 * parts));
  if (n_in > 0 && !given) {
    const int ppr = cinp / 8;
    const long long n_pieces = n_in * ppr;
    if (parts == 2)
      SCN_LAUNCH(k_tile_split<2>, (unsigned)ceil_div(n_pieces, 256), 256, 0, stream, in, split, n_pieces, cin, ppr, SP, pre_scale, pre_shift, pre_leak, in_b, planes_a);
    else
      SCN_LAUNCH(k_tile_split<1>, (unsigned)ceil_div(n_pieces, 256), 256, 0, stream, in, split, n_pieces, cin, ppr, SP, pre_scale, pre_shift, pre_leak, in_b, planes_a);
  }

  TileParams P{};
  P.in_split = given ? (const unsigned char *)rows.in : split;
  P.out_sp = slice_planes(terms, cout);
  unsigned char *out_split = rows.out && cout % P.out_sp == 0 ? (unsigned char *)rows.out : nullptr;
  P.row_bytes = (long long)cinp * 2 * parts;
  P.n_in = n_in;
  P.out = out;
  P.n_out = n_out;
  P.cout = cout;
  P.coutp = coutp;
  P.wprep = (const unsigned char *)wi.ptr;
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
  P.n_tiles = ord.n_tiles;
  P.flags = flags;
  P.drop = g_drop_arrival;
  g_drop_arrival = 0;
  const double w_bytes = (double)coutp * SP * 2 * parts, a_bytes = kRows * SP * 2.0 * parts;
  const char *e = getenv("SCN_TILE_SPLIT");
  P.n_split = e ? std::max(1, atoi(e)) : split_parts(P.n_tiles, ord.one_offset ? 1 : K, n_slices, (a_bytes + w_bytes) / 32.0, cout, n_sm);
  P.out_split = P.n_split > 1 ? nullptr : out_split;
  if (P.n_split > 1) SCN_TRY(tmp.get(&P.out, (size_t)P.n_split * P.n_tiles * kRows * cout * sizeof(float)));
  const auto launch = terms == 3 ? (SP == 32 ? launch_tile<3, 32> : launch_tile<3, 16>) : (SP == 64 ? launch_tile<1, 64> : launch_tile<1, 32>);
  SCN_TRY(launch(P, n_sm, dev, stream));
  if (P.n_split > 1)
    SCN_TRY(sum_partial_tiles(P.out, P.n_split, P.n_tiles * kRows, cout, ord.order, n_out, bias, bn_scale, bn_shift, leak, out,
                              stream, out_split, P.out_sp, parts));
  if (out_split) split_rows_written();
  return SCN_OK;
}

}  // namespace scn
