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
//   * A step's work is small beside the barriers around it, so what bounds it is the longest chain of any one role: 224 to 384 cycles
//     of tensor instructions, 336 (32 -> 32 planes: 20 KB written, 22 read) to 576 (128 -> 128) cycles of shared memory at 128
//     bytes; L2 gives 75 bytes per cycle and SM to 16-byte cp.async gathers of rows that lie in it, a step takes 39 to 58.  Every
//     wait, load and store of shared memory stands 100 to 200 cycles behind the copies.  With a thread of its own for the
//     weights (two waits, a load, an arrival and the copy per step: 1 050 cycles) and instructions issued inside a branch of
//     one lane (descriptors moved into uniform registers one by one: 135 cycles per four instructions, 38 with a predicate) the
//     same tiles took, 8 rooms: 32 -> 32 planes 252 us, now 198; 64 -> 64 144, 128; 96 -> 96 98, 84; 128 -> 128 82, 66;
//     224 -> 224 on 1.4 k rows 22.6, 17.6; 4-D 64 -> 64 bf16 774, 643.  Now, 200 k rows: tensor pipe active 22, 44, 57, 76 % for 32,
//     64, 96, 128 planes, shared memory banks 23 + 17 to 34 + 25 % (read + written), issue slots 55, 52, 40, 39 %.
//
// Roles (14 warps, one or two CTAs per SM, persistent).  A step is one filter offset of one tile and SP input planes; the
// steps of a CTA are numbered through all its tiles and step n uses stage n % n_stages of one ring.
//   entries     one thread: a record per tile (steps, where its rows go) for the roles below, then a slot per filter offset with
//               a rule, the input row of every tile row, one 512-byte bulk copy from the packed table; up to kSlots offsets ahead
//   producers   8 warps, four to a step: 32 rows each by 16-byte cp.async pieces straight into the swizzled operand layout,
//               zero fill where a row has no rule; the barrier arrival happens when a lane's copies have landed.  A warp has
//               the entries of its next step in registers before the stage is free, which also gives the slot back early.
//               The first lane of a step's warps also orders its weights, one bulk copy.  (One warp per step: 2 000
//               cycles from the first copy to the last, during which the stage waits.)
//   MMA         one warp
//   epilogue    4 warps: tcgen05.ld (a lane holds a row) -> shared memory, 16 planes at a time -> bias -> optional
//               BatchNorm scale / shift / leaky ReLU -> 16-byte stores, four lanes per row.  A CTA's last item is stored by the
//               producers as well, a third of the columns for every four warps: 224 planes on 1.4 k rows 19.6 us, 18.2 (with the
//               entries' first loads made before the CTA is set up).  (Stored straight from the TMEM
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
constexpr int kProdWarps = 8, kProdGroups = kProdWarps / kStepWarps;
constexpr int kMma = kProdWarps + 4, kEntries = kMma + 1;
constexpr int kThreads = (kProdWarps + 6) * 32;
constexpr int kStoreSets = 1 + kProdGroups;  // of four warps that store a CTA's last item
constexpr int kSlots = 8;       // offsets the entries run ahead; even, so that a producing warp comes by every slot or every second
constexpr int kMaxStages = 12;
constexpr int kBarriers = 2 * kMaxStages + 2 * kSlots + 8 + 2 * kRecords;
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
  int n_split, per_tile;      // parts of a tile's offsets; items of a tile (the same)
  unsigned char *out_split;  // (optional, n_split 1) the result once more as split rows, slices of out_sp planes
  int out_sp;
  int drop;         // test hook: leave out one barrier arrival of the first CTA
  int *flags;
};

template <int TERMS, int SP>
struct TileShape {
  static constexpr int PARTS = TERMS == 3 ? 2 : 1;
  static constexpr int PP = SP * 2 * PARTS / 16;      // 16-byte pieces per row and step
  static constexpr int NI = 32 / (32 / PP);           // copy instructions per step and lane: a warp has 32 rows of a step
  static constexpr unsigned ROW = PP * 16;            // bytes of a row in a stage: 128 or 64
  static constexpr unsigned A_BYTES = kRows * ROW;
  static_assert(PP == 8 || PP == 4, "a row of a step is 128 or 64 bytes");
};

// control block behind the ring
struct Ctl {
  unsigned long long full[kMaxStages], empty[kMaxStages];  // rows and weights landed; MMAs done
  unsigned long long s_full[kSlots], s_empty[kSlots], acc_full[4], acc_empty[4];
  unsigned long long r_full[kRecords], r_empty[kRecords];
  ItemRecord record[kRecords];
  int total_steps;     // of the CTA, when the slots end
  int slot_k[kSlots];  // filter offset of the slot; -1: no more work; kNoRules: offset 0 with rows of zeros
  OrderedCopies ordered;
  unsigned tmem;
  int abort;
};

// Columns first, first + step, ..., 16 at a time, of the 32 rows that lanes of `quad` hold: tensor memory -> shared memory -> bias
// -> BatchNorm -> the result (and its split form), four lanes per row.  `base`: the accumulator at this quarter of the lanes.
template <int PARTS, bool OUT_SPLIT>
__device__ __forceinline__ void store_columns(const TileParams &P, bool joint, unsigned base, const ItemRecord &R, int orow, int quad,
                                              int lane, float4 *my_epi, int first, int step) {
  const int nc = P.cout;
  // where rows lane / 4, + 8, + 16, + 24 of the warp go: rows of the result, or of the partial sums
  int to[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    to[i] = __shfl_sync(0xffffffffu, orow, i * 8 + (lane >> 2));
    if (!OUT_SPLIT && P.n_split > 1 && to[i] >= 0) to[i] = (R.part * (int)P.n_tiles + R.tile) * kRows + quad * 32 + i * 8 + (lane >> 2);
  }
  for (int c0 = first; c0 < nc; c0 += step) {
#pragma unroll
    for (int half = 0; half < 16; half += 8) {
      unsigned a[8], b[8];
      tmem_ld8_nowait(base + c0 + half, a);
      if (joint) tmem_ld8_nowait(base + P.coutp + c0 + half, b);
      tmem_wait_ld();
#pragma unroll
      for (int e = 0; e < 8; e += 4) {
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
      float4 vs[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = i * 8 + (lane >> 2);
        vs[i] = my_epi[row * 4 + ((lane & 3) ^ ((row >> 1) & 3))];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float4 v = vs[i];
        if (finish && P.bias) v.x += bias.x, v.y += bias.y, v.z += bias.z, v.w += bias.w;
        if (finish && P.bn_scale) {  // separate multiply and add, as the stand-alone BatchNorm kernel rounds them
          v.x = __fadd_rn(__fmul_rn(v.x, sc.x), sh.x), v.y = __fadd_rn(__fmul_rn(v.y, sc.y), sh.y);
          v.z = __fadd_rn(__fmul_rn(v.z, sc.z), sh.z), v.w = __fadd_rn(__fmul_rn(v.w, sc.w), sh.w);
          v.x *= v.x > 0.f ? 1.f : P.leak, v.y *= v.y > 0.f ? 1.f : P.leak;
          v.z *= v.z > 0.f ? 1.f : P.leak, v.w *= v.w > 0.f ? 1.f : P.leak;
        }
        if (to[i] < 0) continue;
        *reinterpret_cast<float4 *>(P.out + (long long)to[i] * nc + c) = v;
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

  if (tid < kBarriers) {  // a thread per barrier, in the order of Ctl
    const int i = tid - 2 * kMaxStages, j = i - 2 * kSlots;
    const unsigned arrivals = tid < kMaxStages ? kStepWarps * 32 + 1  // full: the lanes of the producing warps, and the weights
                              : i < kSlots     ? 1                    // empty, s_full
                              : j < 0          ? kStepWarps * min(P.n_slices, kProdGroups)  // s_empty: the producing warps that come by
                              : j < 4          ? 1                                          // acc_full
                              : j < 8          ? 4                                          // acc_empty
                              : j < 8 + kRecords ? 1                                        // r_full
                                                 : 4 + 1;  // r_empty: the epilogue's warps and the issuing one
    mbar_init(&C.full[0] + tid, arrivals);
    if (tid == 0) C.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  Tiles<TileParams> tiles;
  if (tid == kEntries * 32) tiles.start(P);  // (on its way while tensor memory is had)
  if (warp == kMma) tmem_alloc(&C.tmem, (unsigned)P.tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = C.tmem;
  volatile int *abort = &C.abort;
  const long long my_items = items_here(P.n_items);  // (the grid has at most n_items CTAs)

  if (warp < kProdWarps) {
    // ==================================== producers =============================================
    // Group g of four warps takes the steps g, g + 2, ...; a warp copies 32 rows of a step, a lane one 16-byte piece of the
    // rows q NI .. q NI + NI - 1 of them.  The input rows of the next step are in registers before its stage is free.  A warp leaves
    // as a whole: what its lanes do together has no limit to its wait for one that has gone.
    const int j = lane % PP, q = lane / PP, group = warp / kStepWarps, row0 = warp % kStepWarps * 32 + q * NI;
    // (ROW 128: rows come in eights, chunk j of row r is stored at j ^ (r & 7); ROW 64: in fours, at j ^ ((r >> 1) & 3))
    const unsigned lane_dst = smem0 + (unsigned)row0 * Shape::ROW + (unsigned)((PP == 8 ? j : j ^ (q & 1) * 2) * 16);
    const int d_slot = kProdGroups / P.n_slices, d_slice = kProdGroups % P.n_slices;
    int slot = group / P.n_slices, slice = group % P.n_slices, st = group, par = 1;  // (n_stages is at least kProdGroups)
    const bool brings_weights = warp % kStepWarps == 0 && lane == 0;
    int slot_k = 0, filled = 0;
    bool ok = true, bad = false, fresh = true;
    const unsigned char *const col = P.in_split + j * 16;
    int rows[NI];
    for (;;) {
      if (fresh) {
        const int si = slot % kSlots;
        // (A warp comes by every slot, or by every second one with one slice: it has seen the slot kSlots before this one
        // filled, so the parity cannot be that of an earlier round.)
        ok = mbar_wait_warp(&C.s_full[si], (slot / kSlots) & 1, abort);
        if (!ok) break;
        slot_k = C.slot_k[si];
        if (slot_k < 0) break;
        const int4 *ent = reinterpret_cast<const int4 *>(entries + si * kRows + row0);
#pragma unroll
        for (int i = 0; i < NI; i += 4) {
          const int4 e4 = ent[i / 4];
          rows[i] = e4.x, rows[i + 1] = e4.y, rows[i + 2] = e4.z, rows[i + 3] = e4.w;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&C.s_empty[si]);
#pragma unroll
        for (int i = 0; i < NI; ++i) {
          if (slot_k == kNoRules) rows[i] = -1;
          bad |= rows[i] >= (int)P.n_in;
        }
      }
      ok = mbar_wait_warp(&C.empty[st], par, abort);  // (the first round passes)
      if (!ok) break;
      const unsigned dst = lane_dst + (unsigned)st * stage_bytes;
      if (brings_weights && !(P.drop && blockIdx.x == 0 && group == 0 && filled == 0)) {
        const unsigned char *w = P.wprep + ((size_t)(slot_k == kNoRules ? 0 : slot_k) * P.n_slices + slice) * w_bytes;
        mbar_expect_tx(&C.full[st], w_bytes);
        bulk_copy_g2s(smem0 + (unsigned)st * stage_bytes + Shape::A_BYTES, w, w_bytes, &C.full[st]);
      }
      ++filled;
      const unsigned char *src = col + slice * (SP * 2 * PARTS);
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const bool hit = (unsigned)rows[i] < (unsigned)P.n_in;
        const unsigned swizzle = (PP == 8 ? i & 7 : i >> 1 & 3) * 16;
        cp_async16((dst ^ swizzle) + i * Shape::ROW, src + (size_t)(unsigned)(hit ? rows[i] : 0) * P.row_bytes, hit ? 16u : 0u);
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
    if (!ok) {
      *abort = 1;
    } else if (!__any_sync(0xffffffffu, *abort != 0)) {
      // The CTA's last item: these warps store two thirds of its columns, through the ring, which nothing reads any more when
      // the last step has been consumed.  (The step before it first, whose parity cannot be an earlier round's: this
      // warp has seen the consumption of the one n_stages before either.)
      const int last = (int)my_items - 1, n = C.total_steps, quad = warp & 3;
      const ItemRecord R = C.record[last % kRecords];
      const int orow = __ldg(P.order + (long long)R.tile * kRows + quad * 32 + lane);
      if ((n < 2 || mbar_wait_warp(&C.empty[(n - 2) % P.n_stages], ((n - 2) / P.n_stages) & 1, abort)) &&
          mbar_wait_warp(&C.empty[(n - 1) % P.n_stages], ((n - 1) / P.n_stages) & 1, abort)) {
        tc_fence_after();
        store_columns<PARTS, OUT_SPLIT>(P, joint, tmem + ((unsigned)(quad * 32) << 16) + (unsigned)(last % n_acc * dcols), R, orow, quad,
                                        lane, reinterpret_cast<float4 *>(smem + warp * kEpiBytes), 16 * (1 + group), 16 * kStoreSets);
        tc_fence_before();
      } else {
        *abort = 1;
      }
    }
  } else if (warp == kMma) {
    // ==================================== MMA issue =============================================
    // The whole warp runs the loop and one elected lane issues, by a predicate (mma_bf16_if).
    const unsigned id_all = tile_idesc(joint ? 2 * P.coutp : P.coutp), id_one = tile_idesc(P.coutp);
    const unsigned long long a_desc = rows_desc<Shape::ROW>(smem0, 0);
    const unsigned long long w_desc = smem_desc(smem0 + Shape::A_BYTES, 128, SP / 8 * 128);
    const unsigned a_hi = (unsigned)(a_desc >> 32), w_hi = (unsigned)(w_desc >> 32);
    const unsigned a0 = (unsigned)a_desc, w0 = (unsigned)w_desc;
    const unsigned stage_step = stage_bytes >> 4, wm_step = w_part >> 4;
    const int items = (int)my_items, n_stages = P.n_stages, coutp = P.coutp;
    int st = 0, par = 0, buf = 0, buf_par = 1;
    unsigned d = tmem;
    bool ok = true;
    const unsigned lead = elect_one() ? 1u : 0u;
    bool ready = false;  // the stage at hand, looked at while the instructions of the one before it were issued
    for (int i = 0; i < items && ok; ++i) {
      const int ri = i % kRecords;
      if (!mbar_wait_warp(&C.r_full[ri], (i / kRecords) & 1)) {
        ok = false;
        break;
      }
      const int steps = __reduce_max_sync(0xffffffffu, C.record[ri].steps);
      if (lead) mbar_arrive(&C.r_empty[ri]);
      // the item's accumulator must have been drained
      if (!mbar_wait_warp(&C.acc_empty[buf], buf_par) || __any_sync(0xffffffffu, *abort != 0)) {
        ok = false;
        break;
      }
      for (int s = 0; s < steps; ++s) {
        if (!ready && !mbar_wait_warp(&C.full[st], par)) {
          ok = false;
          break;
        }
        const int st1 = st + 1 == n_stages ? 0 : st + 1, par1 = st1 ? par : par ^ 1;
        const unsigned seen = mbar_test(&C.full[st1], par1);
        // order the copied rows (acquired through the barrier) before the tensor core's async-proxy reads; done
        // here, not by the producers: their fence would wait for the copies they have just started
        fence_proxy_async_smem();
        tc_fence_after();
        const unsigned at = (unsigned)st * stage_step;
#pragma unroll
        for (int jj = 0; jj < SP / 16; ++jj) {
          const unsigned ah = a0 + at + jj * 2, am = ah + SP / 8, wh = w0 + at + jj * 16;
          if (jj == 0) mma_bf16_if(lead, d, ah, a_hi, wh, w_hi, joint ? id_all : id_one, (unsigned)s);
          else mma_bf16_acc_if(lead, d, ah, a_hi, wh, w_hi, joint ? id_all : id_one);
          if (TERMS == 3) {
            if (joint) {
              mma_bf16_acc_if(lead, d + coutp, am, a_hi, wh, w_hi, id_one);
            } else {
              mma_bf16_acc_if(lead, d, ah, a_hi, wh + wm_step, w_hi, id_one);
              mma_bf16_acc_if(lead, d, am, a_hi, wh, w_hi, id_one);
            }
          }
        }
        tc_commit_if(lead, &C.empty[st]);
        if (s == steps - 1) tc_commit_if(lead, &C.acc_full[buf]);
        st = st1, par = par1;
        ready = __all_sync(0xffffffffu, seen != 0);
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
      for (long long it = 0; it < my_items && ok; ++it) {
        unsigned u[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) u[w] = tiles.mask[w];
        const int tile = tiles.tile, part = P.n_split == 1 ? 0 : (int)item_of(it) % P.n_split;
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
        C.record[ri] = ItemRecord{max(1, offsets) * P.n_slices, tile, part, tiles.tile};
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
      // every producing warp finds its next step in a slot that ends it
      const int ends = (kProdGroups - 1) / P.n_slices + 1;
      C.total_steps = slot * P.n_slices;
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
  } else {
    // ==================================== epilogue ==============================================
    const int quad = warp & 3;
    float4 *my_epi = reinterpret_cast<float4 *>(epi + quad * kEpiBytes);
    int buf = 0, buf_par = 0;
    int next_orow = 0;  // this lane's row of the next item: asked for an item ahead
    for (int it = 0; it < (int)my_items; ++it) {
      const int ri = it % kRecords;
      if (!mbar_wait_warp(&C.r_full[ri], (it / kRecords) & 1, abort)) {
        *abort = 1;
        break;
      }
      const ItemRecord R = C.record[ri];  // (each lane has seen the phase: a shuffle of one lane's answer orders no memory)
      __syncwarp();
      if (lane == 0) mbar_arrive(&C.r_empty[ri]);
      const int orow = it ? next_orow : __ldg(P.order + (long long)R.tile * kRows + quad * 32 + lane);
      next_orow = __ldg(P.order + (long long)R.next_tile * kRows + quad * 32 + lane);
      if (!mbar_wait_warp(&C.acc_full[buf], buf_par, abort)) {
        *abort = 1;
        break;
      }
      tc_fence_after();
      store_columns<PARTS, OUT_SPLIT>(P, joint, tmem + ((unsigned)(quad * 32) << 16) + (unsigned)(buf * dcols), R, orow, quad, lane, my_epi,
                                      0, it == (int)my_items - 1 ? 16 * kStoreSets : 16);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&C.acc_empty[buf]);
      if (++buf == n_acc) buf = 0, buf_par ^= 1;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort) {
    if (tid == 0) atomicOr(P.flags, FLAG_TC_TIMEOUT);
    land_copies(C, P.n_stages, kProdGroups);
  }
  __syncwarp();
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
  const long long step = n_pos * cout4;
  // the first four parts and the row on their way together (a place without a row has room for parts as well)
  float4 v[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) v[p] = p < n_split ? __ldg(partial + p * step + i) : make_float4(0.f, 0.f, 0.f, 0.f);
  const long long r = order ? __ldg(order + i / cout4) : i / cout4;
  if (r < 0 || r >= n_out) return;
  float4 q = v[0];
#pragma unroll
  for (int p = 1; p < 4; ++p)
    if (p < n_split) q.x += v[p].x, q.y += v[p].y, q.z += v[p].z, q.w += v[p].w;
#pragma unroll 4
  for (int p = 4; p < n_split; ++p) {
    const float4 a = __ldg(partial + p * step + i);
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
  P.per_tile = P.n_split;
  P.n_items = P.n_tiles * P.per_tile;
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
// plus, with more than one part, the partial sums' traffic and the second launch.  In SM cycles: a step counts as its bytes (rows and
// weights) at 32 per cycle, an item's fill and drain as 2 500, for one CTA per SM.  The constants are empirical and older than the
// kernel's present form, whose steps take 39 to 58 bytes per cycle.  What they choose, measured against 1 to 16 parts on 48 layers of
// U-Nets, 40 to 57 k rows, 32 to 448 planes: within 5 % of the best on 42; 64 -> 64 planes on 10.7 k rows 20.8 us (three parts: 16.1);
// 160 -> 160 and 320 -> 160 on 22 k 61 and 107 (57 and 101); three strided layers 11 to 13 (one microsecond less).
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
  P.n_split = e ? std::max(1, std::min<int>(atoi(e), (int)((1ll << 31) / (P.n_tiles * kRows) - 1))) : split_parts(P.n_tiles, ord.one_offset ? 1 : K, n_slices, (a_bytes + w_bytes) / 32.0, cout, n_sm);
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
