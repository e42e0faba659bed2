// Weight gradients on tcgen05 tensor cores over mask-sorted row tiles.
//
//     d_W[k] = sum over the rules (i, o) of offset k of in[i]^T d_out[o]        (CUDA/Convolution.cu dW kernels)
//
// The rows of a tile (row_order.cu) share their filter offsets, so for one tile and one offset the rules are 128 rows of
// the matrix on the table's own side (T: d_out, or `in` for a Deconvolution) against 128 gathered rows of the other (G).
// The contraction runs over the rules: both operands are staged as they lie in memory, one rule per 128-byte row with its
// planes contiguous, and read M- / N-major by the MMA -- no transposition anywhere.
//
//   arithmetic  x = h + m + l, three bf16 parts that hold all 24 bits of x; every product of the parts but m l, l m and
//               l l (2^-24 of a product) is summed in fp32.  The parts of T are lanes of one accumulator (M = 128: h and m of 64 planes, or h, m and l of 32),
//               those of G its columns, and the blocks are added when the sums are done; the products with an l go where
//               those with an m go.  The tensor core truncates its running sum at every instruction, half a unit of 2^-24 on
//               average: a CTA takes at most kMaxTiles tiles, 8 instructions each for the sums of h h (up to 24 for the
//               others, which are 2^-8 as large), before its sums are added in fp32.
//   split       The accumulators of a CTA stay in TMEM from its first rule to its last: 5 filter offsets x 96 columns (32
//               gathered planes) or 4 x 128 (64).  A CTA is one such group of offsets, one pair of plane blocks and every
//               n_chunks-th tile; the chunks' sums are added in order (k_sum_chunks), so the result does not depend on
//               timing.  The partial sums of a launch take at most kMostPartial bytes; a layer with more chunks than fit
//               is done in several launches, each adding to the sum of those before.
//   jobs        One thread walks the tiles: a job is the T rows of a tile or the G rows of one of its offsets, a slot of a
//               ring with the 128 row numbers (a 512-byte bulk copy) and what they are for.
//   staging     8 warps copy rows of the split matrices (k_dweight_split, once per call) with 16-byte cp.async straight into
//               the swizzled operand rows.  The G rows go in pieces of 32 rows to one stage and one warp each, so that
//               a warp's chain of waits is spread over eight pieces (with every job spread over all warps it was 2 500 cycles
//               per job); a tile's T rows are staged once for all the group's offsets, 16 rows by each warp.  (Splitting
//               gathered fp32 rows on their way through the registers moves a third fewer bytes, but at 55 instructions per
//               16 bytes the warps could not keep up: 5 600 cycles per piece.)
//   MMA         two warps, a job's 128 rules at a time.  An instruction's issue takes as long as the tensor core does, and what
//               a warp spends on barriers and its next job (some 800 cycles for 1 408 of instructions) came on top: 64 x 96
//               weights on 131 k rows 346 us with one warp that waited for every 32 rules, 311 for 128, 302 with two warps.
//
// Bound by the gather: 48 KB per 128 rules of 64 planes and a share of the tile's own rows, 72 KB in 2 100 cycles, beside
// 1 408 cycles of tensor instructions.
#include <algorithm>
#include <atomic>
#include <utility>

#include "conv_tile.cuh"

namespace scn {

__global__ void k_sum_chunks(const float *__restrict__ partial, int chunks, long long n, float *__restrict__ out, bool add);

namespace {

constexpr int kRows = kOrderTile;
constexpr int kLoadWarps = 8;
constexpr int kMmaWarps = 2, kMma = kLoadWarps, kJobs = kMma + kMmaWarps;
constexpr int kThreads = (kJobs + 1) * 32;
constexpr int kSlots = 8;           // jobs ahead
constexpr int kMaxTiles = 48;       // tiles of a CTA
constexpr long long kMostPartial = 256ll << 20;
constexpr int kAtom = kRows * 128;  // 128 rules x 64 elements

template <int PT, int PG>
struct DwTile {
  static constexpr int T_ATOMS = PT == 64 ? 3 : 2;  // h, m, l, or (h m), (l 0)
  static constexpr int G_ATOMS = PG == 64 ? 3 : 2;
  static constexpr int T_PIECE = kRows / kLoadWarps;                             // rows of a warp
  static constexpr int G_PIECE = 32, PIECES = kRows / G_PIECE;                   // rows of a stage, stages of a job
  static constexpr int T_BYTES = T_ATOMS * kAtom, G_ATOM = G_PIECE * 128, G_BYTES = G_ATOMS * G_ATOM;
  // One stage per loading warp: a warp that comes back to its stage has seen the consumption of its last piece but one,
  // so that the parity it waits for cannot be one of an earlier round.
  static constexpr int STAGES = kLoadWarps;
  static_assert(STAGES == 2 * PIECES, "two jobs' rows");
  static constexpr int COLS = PG == 64 ? 128 : 96;  // accumulator columns of an offset
  static constexpr int OFFSETS = 512 / COLS;
  static constexpr int ZERO = 2048;                 // 16 rules of zeros: what follows l in its operand
  static constexpr size_t SMEM = 2 * T_BYTES + STAGES * G_BYTES + ZERO + kSlots * kRows * sizeof(int) + 1024;
};

struct DwParams {
  const unsigned char *t_rows, *g_rows;  // split: the table's side (rows order[.]) and the gathered side (rows packed[.])
  int t_planes, g_planes;
  long long n_t, n_g;
  const int *order, *packed, *by_work;
  const unsigned *tile_bits;
  int words, K, n_groups, n_chunks, first_chunk, blocks_g;  // (first_chunk: of the launch)
  unsigned group_bits[32][4];  // the offsets of a group, ascending, are the bits of its mask
  long long n_tiles;
  int t_is_out;    // T is d_out (else `in`, the operator ran the table backwards)
  int cin, cout;
  float *partial;  // [chunks of the launch][K][cin][cout]
  int *flags;
};

// 64 elements x 8 rules per 1 KB, rows of 128 bytes, 16-byte chunk c of rule r at c ^ (r & 7)
__device__ __forceinline__ unsigned planes_desc_lo(unsigned addr, unsigned next_atom) {
  return ((addr >> 4) & 0x3FFF) | (((next_atom >> 4) & 0x3FFF) << 16);
}
constexpr unsigned kDescHi = (1024 >> 4) | (1u << 14) | (2u << 29);

// both operands M- / N-major, bf16, fp32 sums, M = 128
constexpr unsigned idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((unsigned)(n >> 3) << 17) | ((unsigned)(kRows >> 4) << 24);
}

__device__ __forceinline__ void split3(float a, float b, unsigned &h, unsigned &m, unsigned &l) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  h = *reinterpret_cast<unsigned *>(&v);
  const float ra = a - __uint_as_float(h << 16), rb = b - __uint_as_float(h & 0xFFFF0000u);
  v = __floats2bfloat162_rn(ra, rb);
  m = *reinterpret_cast<unsigned *>(&v);
  v = __floats2bfloat162_rn(ra - __uint_as_float(m << 16), rb - __uint_as_float(m & 0xFFFF0000u));
  l = *reinterpret_cast<unsigned *>(&v);
}

// Bytes of a split row of 8 `pieces` planes in blocks of B: 6 per plane, a row of 32 planes padded to two whole lines (its
// h and m are one; at 192 bytes every other row's lay across two).
__host__ __device__ inline long long split_row_bytes(int pieces, int B) { return B == 32 ? 256 : pieces * 48; }

// x [n][planes] -> per row and block of B planes [B h | B m | B l], planes past the end zero (B 32: one block).  One thread
// per 8 planes.  Bound by HBM: 32 bytes in, 48 out.
__global__ void __launch_bounds__(256)
k_dweight_split(const float *__restrict__ x, unsigned char *__restrict__ out, long long n_pieces, int planes, int per_row, int B) {
  SCN_GRID_WAIT();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_pieces) return;
  const long long row = i / per_row;
  const int c = (int)(i - row * per_row) * 8;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
  if (c < planes) a = __ldg(reinterpret_cast<const float4 *>(x + row * planes + c));
  if (c + 4 < planes) b = __ldg(reinterpret_cast<const float4 *>(x + row * planes + c + 4));
  uint4 h, m, l;
  split3(a.x, a.y, h.x, m.x, l.x);
  split3(a.z, a.w, h.y, m.y, l.y);
  split3(b.x, b.y, h.z, m.z, l.z);
  split3(b.z, b.w, h.w, m.w, l.w);
  uint4 *q = reinterpret_cast<uint4 *>(out + row * split_row_bytes(per_row, B) + c / B * B * 6 + c % B * 2);
  q[0] = h;
  q[B / 8] = m;
  q[B / 4] = l;
}

// N rows of B planes (row numbers in shared memory, -1 or out of range: zeros) into operand rows, 64 elements per atom
template <int B, int N>
__device__ __forceinline__ bool copy_rows(unsigned dst, int atom, const int *rows, const unsigned char *src, long long row_bytes,
                                          int n_rows, int lane) {
  bool bad = false;
  const int q = lane >> 3, c = lane & 7;  // four rows of eight pieces
#pragma unroll
  for (int i = 0; i < N / 4; ++i) {
    const int r = i * 4 + q, e = rows[r];
    const bool hit = (unsigned)e < (unsigned)n_rows;
    bad |= e >= n_rows;
    const unsigned char *p = src + (long long)(hit ? e : 0) * row_bytes + c * 16;
    const unsigned d = dst + r * 128 + (unsigned)((c ^ (r & 7)) * 16), bytes = hit ? 16u : 0u;
    cp_async16(d, p, bytes);
    if (B == 64) {
      cp_async16(d + atom, p + 128, bytes);
      cp_async16(d + 2 * atom, p + 256, bytes);
    }
  }
  if (B == 32) {  // l: four pieces of eight rows
#pragma unroll
    for (int i = 0; i < N / 8; ++i) {
      const int r = i * 8 + (lane >> 2), e = rows[r], cl = lane & 3;
      const bool hit = (unsigned)e < (unsigned)n_rows;
      cp_async16(dst + atom + r * 128 + (unsigned)((cl ^ (r & 7)) * 16), src + (long long)(hit ? e : 0) * row_bytes + 128 + cl * 16, hit ? 16u : 0u);
    }
  }
  return bad;
}

constexpr int kTRows = 100, kEnd = 101;

struct Ctl {
  unsigned long long full[2], empty[2], t_full[2], t_empty[2], s_full[kSlots], s_empty[kSlots], done;
  int job[kSlots];  // index of the offset in the group; kTRows; kEnd
  unsigned tmem, used;
  int abort, slots;  // slots: filled by the jobs
};

template <int PT, int PG>
__global__ void __launch_bounds__(kThreads, 1) k_dweight_tile(const __grid_constant__ DwParams P) {
  SCN_GRID_WAIT();
  using S = DwTile<PT, PG>;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ Ctl C;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int group = blockIdx.x, chunk = P.first_chunk + blockIdx.y, pair = blockIdx.z;
  const int t0 = pair / P.blocks_g * PT, g0 = pair % P.blocks_g * PG;  // first planes of the pair
  const int n_off = __popc(P.group_bits[group][0]) + __popc(P.group_bits[group][1]) + __popc(P.group_bits[group][2]) +
                    __popc(P.group_bits[group][3]);
  const unsigned smem0 = (smem_u32(smem) + 1023u) & ~1023u;
  unsigned char *base = smem + (smem0 - smem_u32(smem));
  const unsigned g_at = 2 * S::T_BYTES, zero_at = g_at + S::STAGES * S::G_BYTES;
  int *rows = reinterpret_cast<int *>(base + zero_at + S::ZERO);  // [kSlots][128]

  // zeros where the operands have elements nobody writes
  if (PT == 32)
    for (int i = tid; i < 2 * S::T_BYTES / 16; i += kThreads) reinterpret_cast<uint4 *>(base)[i] = make_uint4(0, 0, 0, 0);
  for (int i = tid; i < S::ZERO / 16; i += kThreads) reinterpret_cast<uint4 *>(base + zero_at)[i] = make_uint4(0, 0, 0, 0);
  fence_proxy_async_smem();
  if (tid == 0) {
    for (int i = 0; i < S::STAGES / S::PIECES; ++i) {
      mbar_init(&C.full[i], 32 * S::PIECES);  // the lanes of the copying warps
      mbar_init(&C.empty[i], kMmaWarps);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&C.t_full[i], kLoadWarps * 32);
      mbar_init(&C.t_empty[i], kMmaWarps);
    }
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&C.s_full[i], 1);
      mbar_init(&C.s_empty[i], kLoadWarps + kMmaWarps);
    }
    mbar_init(&C.done, kMmaWarps);
    C.abort = 0;
    C.used = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMma) tmem_alloc(&C.tmem, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = C.tmem;
  volatile int *abort = &C.abort;

  if (warp < kLoadWarps) {
    // ==================================== rows ==================================================
    const long long t_bytes = split_row_bytes((P.t_planes + PT - 1) / PT * (PT / 8), PT), g_bytes = split_row_bytes((P.g_planes + PG - 1) / PG * (PG / 8), PG);
    const unsigned char *t_src = P.t_rows + t0 * 6, *g_src = P.g_rows + g0 * 6;
    const unsigned t_dst = smem0 + warp * (S::T_PIECE * 128), g_dst = smem0 + g_at + warp * S::G_BYTES;  // piece g: stage g % 8
    bool bad = false, ok = true;
    int slot = 0, s_par = 0, n_g = 0, n_t = 0;  // of the slot: first G piece, tile
    for (;;) {
      ok = mbar_wait_warp(&C.s_full[slot], s_par, abort);
      if (!ok) break;
      const int job = C.job[slot];
      if (job == kEnd) break;
      const int *row = rows + slot * kRows;
      if (job == kTRows) {
        const int tb = n_t & 1;
        ok = mbar_wait_warp(&C.t_empty[tb], (unsigned)((n_t >> 1) + 1) & 1, abort);
        if (!ok) break;
        bad |= copy_rows<PT, S::T_PIECE>(t_dst + tb * S::T_BYTES, kAtom, row + warp * S::T_PIECE, t_src, t_bytes, (int)P.n_t, lane);
        cp_async_arrive(&C.t_full[tb]);
        ++n_t;
      } else {
        const int q = (warp - n_g) & (kLoadWarps - 1);  // the piece of the job that is this warp's
        if (q < S::PIECES) {
          ok = mbar_wait_warp(&C.empty[warp / S::PIECES], (unsigned)((n_g + q) / S::STAGES + 1) & 1, abort);
          if (!ok) break;
          bad |= copy_rows<PG, S::G_PIECE>(g_dst, S::G_ATOM, row + q * S::G_PIECE, g_src, g_bytes, (int)P.n_g, lane);
          cp_async_arrive(&C.full[warp / S::PIECES]);
        }
        n_g += S::PIECES;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&C.s_empty[slot]);
      if (++slot == kSlots) slot = 0, s_par ^= 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");  // they must land before the CTA's shared memory goes away
    if (bad) atomicOr(P.flags, FLAG_BAD_ROW);
    if (!ok) *abort = 1;
  } else if (warp == kJobs) {
    // ==================================== jobs ==================================================
    if (lane == 0) {
      unsigned mine[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) mine[w] = P.group_bits[group][w];
      constexpr int kFetch = 4;  // tiles whose masks are on their way
      unsigned u[kFetch][4];
      long long tile[kFetch];
      // the tiles with the most offsets first, back and forth over the chunks
      auto place = [&](long long it) { return it & 1 ? (it + 1) * P.n_chunks - 1 - chunk : it * P.n_chunks + chunk; };
      auto fetch = [&](int i, long long it) {
        const long long at = place(it);
        tile[i] = at < P.n_tiles ? (P.by_work ? (long long)__ldg(P.by_work + at) : at) : -1;
#pragma unroll
        for (int w = 0; w < 4; ++w) u[i][w] = tile[i] >= 0 && w < P.words ? __ldg(P.tile_bits + tile[i] * P.words + w) : 0u;
      };
      const long long full = P.n_tiles / P.n_chunks, rounds = full + (place(full) < P.n_tiles ? 1 : 0);
#pragma unroll
      for (int i = 0; i < kFetch; ++i) fetch(i, i);
      int n = 0;
      bool ok = true;
      auto put = [&](int job, const int *src) {
        const int si = n % kSlots;
        if (!mbar_wait(&C.s_empty[si], ((n / kSlots) + 1) & 1) || *abort) {
          ok = false;
          return;
        }
        C.job[si] = job;
        if (src) {
          mbar_expect_tx(&C.s_full[si], kRows * 4);
          bulk_copy_g2s(smem_u32(rows + si * kRows), src, kRows * 4, &C.s_full[si]);
        } else {
          mbar_arrive(&C.s_full[si]);
        }
        ++n;
      };
      for (long long it = 0; it < rounds && ok;) {
#pragma unroll
        for (int i = 0; i < kFetch; ++i) {
          if (it >= rounds || !ok) break;
          const long long t = tile[i];
          if ((u[i][0] & mine[0]) | (u[i][1] & mine[1]) | (u[i][2] & mine[2]) | (u[i][3] & mine[3])) {
            put(kTRows, P.order + t * kRows);
            const int *src = P.packed + t * P.K * kRows;
            int before = 0, j = 0;  // offsets of the tile, and of the group, in the words already passed
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              for (unsigned m = u[i][w] & mine[w]; m && ok; m &= m - 1) {
                const int bit = __ffs(m) - 1;
                put(j + __popc(mine[w] & ((1u << bit) - 1u)), src + (before + __popc(u[i][w] & ((1u << bit) - 1u))) * kRows);
              }
              before += __popc(u[i][w]);
              j += __popc(mine[w]);
            }
          }
          fetch(i, it + kFetch);
          ++it;
        }
      }
      if (ok) put(kEnd, nullptr);
      C.slots = n;
      if (!ok) *abort = 1;
    }
    __syncwarp();  // the other lanes must not go ahead: waiting for `done` they would hold up lane 0
  } else {
    // ==================================== MMA issue =============================================
    // Each warp issues the jobs of every second offset of the group: an accumulator belongs to one of them, and what one
    // takes to learn of its next job and to wait for its rows passes while the other's instructions run.  The whole warp runs
    // the loop, one elected lane issues; the job is made warp-uniform by a reduction, so that the descriptors stay in
    // uniform registers.
    const int parity = warp - kMma;
    int slot = 0, s_par = 0, st = 0, par = 0, tb = 1, t_par = 1;  // (the first tile's T rows are buffer 0, parity 0)
    unsigned used = 0;
    bool ok = true, first = true;
    const bool leader = elect_one();
    for (;;) {
      if (!mbar_wait_warp(&C.s_full[slot], s_par) || __any_sync(0xffffffffu, *abort != 0)) {
        ok = false;
        break;
      }
      const int job = __reduce_max_sync(0xffffffffu, C.job[slot]);
      if (lane == 0) mbar_arrive(&C.s_empty[slot]);
      if (++slot == kSlots) slot = 0, s_par ^= 1;
      if (job == kEnd) break;
      if (job == kTRows) {
        if (!first && leader) tc_commit(&C.t_empty[tb]);
        __syncwarp();
        first = false;
        if (++tb == 2) tb = 0, t_par ^= 1;
        if (!mbar_wait_warp(&C.t_full[tb], t_par)) {
          ok = false;
          break;
        }
        continue;
      }
      // (for the other warp's jobs too, and the rows go when both have been here: neither can fall a round behind, or run a
      // round ahead, where a phase's parity is that of another)
      if (!mbar_wait_warp(&C.full[st], par)) {
        ok = false;
        break;
      }
      if ((job & 1) != parity) {
        if (lane == 0) mbar_arrive(&C.empty[st]);
      } else {
        const unsigned a = smem0 + tb * S::T_BYTES, d = tmem + job * S::COLS;
        const unsigned al = a + 2 * kAtom;
        const unsigned A = planes_desc_lo(a, kAtom), AL = planes_desc_lo(al, smem0 + zero_at - al);
        const unsigned B0 = planes_desc_lo(smem0 + g_at + st * (S::PIECES * S::G_BYTES), S::G_ATOM);
        const unsigned acc = (used >> job) & 1u;
        if (leader) {
          // order the stored rows (acquired through the barriers) before the tensor core's async-proxy reads; done here,
          // not by the warps that store: their fence would wait for the loads they have on their way
          fence_proxy_async_smem();
          tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < kRows / 16; ++kk) {
            const unsigned B = B0 + kk / 2 * (S::G_BYTES >> 4) + kk % 2 * 128;  // a piece, and 2 KB further
            if (kk == 0) mma_bf16(d, A, kDescHi, B, kDescHi, idesc(PG == 64 ? 128 : 96), acc);
            else mma_bf16_acc(d, A + kk * 128, kDescHi, B, kDescHi, idesc(PG == 64 ? 128 : 96));
            if (PG == 64) mma_bf16_acc(d + 64, A + kk * 128, kDescHi, B + (2 * S::G_ATOM >> 4), kDescHi, idesc(64));
            // l of T with h of G, zeros behind l: 2 KB further, and the zeros 2 KB nearer
            if (PT == 64) mma_bf16_acc(d + PG, AL + kk * 128 - (unsigned)(kk * 128 << 16), kDescHi, B, kDescHi, idesc(PG));
          }
          tc_commit(&C.empty[st]);
        }
        __syncwarp();
        used |= 1u << job;
      }
      if (++st == S::STAGES / S::PIECES) st = 0, par ^= 1;
    }
    if (!ok) *abort = 1;
    if (leader) {
      atomicOr(&C.used, used);
      tc_commit(&C.done);
    }
    __syncwarp();
  }

  // ==================================== sums ====================================================
  if (!mbar_wait(&C.done, 0)) *abort = 1;
  __syncthreads();
  tc_fence_after();
  float *sh = reinterpret_cast<float *>(base);  // [4 lane quarters][32][PG + 1]: every MMA has been read out of it
  const unsigned used = C.used;
  if (!*abort) {
    unsigned left[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) left[w] = P.group_bits[group][w];
    for (int j = 0; j < n_off; ++j) {
      int k = 0;
#pragma unroll
      for (int w = 3; w >= 0; --w)
        if (left[w]) k = w * 32 + __ffs(left[w]) - 1;
#pragma unroll
      for (int w = 0; w < 4; ++w)
        if (k >> 5 == w) left[w] &= left[w] - 1;
      const bool any = (used >> j) & 1u;
      if (any && warp < 4) {
        const unsigned d = tmem + ((unsigned)(warp * 32) << 16) + j * S::COLS;
#pragma unroll
        for (int c0 = 0; c0 < PG; c0 += 16) {
          unsigned a[16], b[16], c[16];
          tmem_ld16_nowait(d + c0, a);
          tmem_ld16_nowait(d + PG + c0, b);
          if (PG == 32) tmem_ld16_nowait(d + 2 * PG + c0, c);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            float x = __uint_as_float(b[e]);
            if (PG == 32) x += __uint_as_float(c[e]);
            sh[(warp * 32 + lane) * (PG + 1) + c0 + e] = __uint_as_float(a[e]) + x;
          }
        }
        tc_fence_before();
      }
      __syncthreads();
      float *out = P.partial + ((long long)blockIdx.y * P.K + k) * P.cin * P.cout;
      for (int i = tid; i < PT * PG; i += kThreads) {
        const int tp = P.t_is_out ? i % PT : i / PG, gp = P.t_is_out ? i / PT : i % PG;
        if (t0 + tp >= P.t_planes || g0 + gp >= P.g_planes) continue;
        float x = 0.f;
        if (any) {
          const float *q = sh + tp * (PG + 1) + gp;
          if (PT == 64) x = q[0] + q[64 * (PG + 1)];
          else x = q[0] + (q[32 * (PG + 1)] + q[64 * (PG + 1)]);
        }
        if (P.t_is_out) out[(long long)(g0 + gp) * P.cout + t0 + tp] = x;
        else out[(long long)(t0 + tp) * P.cout + g0 + gp] = x;
      }
      __syncthreads();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort) {
    if (tid == 0) atomicOr(P.flags, FLAG_TC_TIMEOUT);
    land_slots(C.s_full, C.slots);
  }
  __syncwarp();
  if (warp == kMma) tmem_dealloc(tmem, 512);
}

template <int PT, int PG>
int launch(DwParams &P, const Rulebook &rb, const float *t_rows, const float *g_rows, float *d_weight, cudaStream_t stream) {
  using S = DwTile<PT, PG>;
  static std::atomic<bool> configured[64];
  int dev = 0;
  SCN_CUDA_CHECK(cudaGetDevice(&dev));
  SCN_REQUIRE(dev >= 0 && dev < 64, SCN_ERR_UNSUPPORTED, "device index %d unsupported", dev);
  if (!configured[dev].load()) {
    SCN_CUDA_CHECK(cudaFuncSetAttribute(k_dweight_tile<PT, PG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM));
    configured[dev].store(true);
  }
  // Groups that weigh about the same.  On surfaces and volumes an offset's rules fall off with the number of dimensions it
  // moves in (about 1, 0.6, 0.3, 0.1 of the rows); the heaviest offset left goes to the lightest group that has room.
  // (Every n_groups-th offset put all nine of a floor's offsets in two groups of six.)
  P.n_groups = (int)ceil_div(P.K, S::OFFSETS);
  std::pair<int, int> by[kOrderMaxOffsets];  // weight (negative, to sort), offset
  for (int k = 0; k < P.K; ++k) {
    int moves = 0, rest = k;
    for (int d = rb.dim - 1; d >= 0; --d) {
      moves += rb.symmetric && rest % rb.filter[d] != rb.filter[d] / 2;
      rest /= (int)rb.filter[d];
    }
    by[k] = {moves == 0 ? -10 : moves == 1 ? -6 : moves == 2 ? -3 : -1, k};
  }
  std::sort(by, by + P.K);
  int load[32] = {0}, size[32] = {0};
  for (int i = 0; i < P.K; ++i) {
    int to = -1;
    for (int g = 0; g < P.n_groups; ++g)
      if (size[g] < S::OFFSETS && (to < 0 || load[g] < load[to])) to = g;
    load[to] -= by[i].first;
    ++size[to];
    P.group_bits[to][by[i].second >> 5] |= 1u << (by[i].second & 31);
  }
  P.blocks_g = (int)ceil_div(P.g_planes, PG);
  const int pairs = (int)ceil_div(P.t_planes, PT) * P.blocks_g;
  // one CTA per SM, in whole waves where the groups and blocks leave room for it
  const long long per_wave = std::max(1, 148 / (P.n_groups * pairs));
  P.n_chunks = (int)std::min<long long>(P.n_tiles, per_wave * ceil_div(P.n_tiles, per_wave * kMaxTiles));
  const long long w_elems = (long long)P.K * P.cin * P.cout;
  Scratch tmp(stream);
  P.partial = d_weight;
  const int at_once = (int)std::min<long long>(P.n_chunks, std::max<long long>(per_wave, kMostPartial / ((long long)sizeof(float) * w_elems)));
  if (P.n_chunks > 1) SCN_TRY(tmp.get(&P.partial, sizeof(float) * (size_t)at_once * w_elems));
  unsigned char *split = nullptr;
  const int t_per = (int)ceil_div(P.t_planes, PT) * PT / 8, g_per = (int)ceil_div(P.g_planes, PG) * PG / 8;
  const size_t t_size = (size_t)(P.n_t * split_row_bytes(t_per, PT)), g_size = (size_t)(P.n_g * split_row_bytes(g_per, PG));
  SCN_TRY(tmp.get(&split, t_size + g_size));
  P.t_rows = split;
  P.g_rows = split + t_size;
  SCN_LAUNCH(k_dweight_split, (unsigned)ceil_div(P.n_t * t_per, 256), 256, 0, stream, t_rows, split, P.n_t * t_per, P.t_planes, t_per, PT);
  SCN_LAUNCH(k_dweight_split, (unsigned)ceil_div(P.n_g * g_per, 256), 256, 0, stream, g_rows, split + t_size, P.n_g * g_per, P.g_planes, g_per, PG);
  for (; P.first_chunk < P.n_chunks; P.first_chunk += at_once) {
    const int here = std::min(at_once, P.n_chunks - P.first_chunk);
    SCN_LAUNCH((k_dweight_tile<PT, PG>), dim3((unsigned)P.n_groups, (unsigned)here, (unsigned)pairs), kThreads, S::SMEM, stream, P);
    if (P.n_chunks > 1)
      SCN_LAUNCH(k_sum_chunks, (unsigned)ceil_div(w_elems, 256), 256, 0, stream, P.partial, here, w_elems, d_weight, P.first_chunk > 0);
  }
  SCN_CUDA_CHECK(cudaGetLastError());
  return SCN_OK;
}

}  // namespace

// Rows of whole 16-byte pieces and more than 32 planes on one side: 32 x 32 weights are half as much work per gathered
// byte, and k_conv_dweight_mma takes as long (278 us on 434 k rows).  Both kernels on the others: 64 x 64 on 119 k rows 230
// and, here, 160 us, 96 x 96 on 49 k 412 and 229, 128 x 128 on 6 k 110 and 79.  Below 2048 rows an order has to be there
// already, and not only because an fp32 convolution has made it.
// Multiples of 32 planes only: the running sums in TMEM cut off where fp32 additions round, 4e-6 of a sum of 100 k products
// of mixed signs and 8e-6 with one sign.  That is no more than these shapes ever had (5e-6 and 1e-5 with truncated tf32 parts);
// the others had plain fp32 sums (9e-7, 1.4e-7), which k_conv_dweight_mma matches.
bool dweight_tile_supported(const float *in, const float *d_out, const Rulebook &rb, int cin, int cout) {
  return cin % 32 == 0 && cout % 32 == 0 && (rb.n_out >= 2048 || (rb.n_out > 0 && rb.order.order && !rb.order.fp32_only)) && std::max(cin, cout) > 32 && rb.n_offsets <= kOrderMaxOffsets &&
         ((uintptr_t)in | (uintptr_t)d_out) % 16 == 0;
}

// rb.order packs the rulebook's own table; swap: the operator ran it backwards (d_out is the gathered side)
int dweight_tile(const float *in, long long rows_in, const float *d_out, long long rows_out, const Rulebook &rb, bool swap, int cin,
                 int cout, float *d_weight, int *flags, cudaStream_t stream) {
  SCN_REQUIRE(rows_in < (1ll << 31) && rows_out < (1ll << 31), SCN_ERR_UNSUPPORTED, "row count above 2^31");
  const RowOrder &ord = rb.order;
  const int K = rb.n_offsets;
  DwParams P{};
  const float *t_rows = swap ? in : d_out, *g_rows = swap ? d_out : in;
  P.t_planes = swap ? cin : cout;
  P.g_planes = swap ? cout : cin;
  P.n_t = swap ? rows_in : rows_out;
  P.n_g = swap ? rows_out : rows_in;
  P.order = ord.order;
  P.packed = ord.packed;
  P.by_work = ord.by_work;
  P.tile_bits = ord.tile_bits;
  P.words = ord.words;
  P.n_tiles = ord.n_tiles;
  P.K = K;
  P.t_is_out = !swap;
  P.cin = cin;
  P.cout = cout;
  P.flags = flags;
  if (P.t_planes <= 32) return launch<32, 64>(P, rb, t_rows, g_rows, d_weight, stream);
  return P.g_planes <= 32 ? launch<64, 32>(P, rb, t_rows, g_rows, d_weight, stream) : launch<64, 64>(P, rb, t_rows, g_rows, d_weight, stream);
}

}  // namespace scn
