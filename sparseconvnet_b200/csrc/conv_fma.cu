// fp32 sparse convolution (fused multiply-adds only) over mask-sorted row tiles: few output planes on many rows, small levels
// and little work; the rest of the fp32 mode runs on tensor cores (conv_six.cu: conv_six_takes has the line and both sides).
//
// Same arithmetic class as k_conv_pipe (conv_pipe.cu) and k_conv_simt (conv_simt.cu; the reference's per-offset gather /
// GEMM / scatter-add is CPU/Convolution.cpp:137-148, CUDA/Convolution.cu:57-233): fp32 products, fp32 sums.  A CTA of 128
// threads owns ROWS rows of one packed tile (row_order.cu) and BN output planes.  Because the rows of a tile share their
// filter offsets, the tile is treated as dense: every thread keeps TM x TN results in registers from the first offset to
// the last, a missing rule is a row of zeros, and there are no pair lists, no accumulator in shared memory and no fold.
// A tile of 128 rows meets 9 to 12 of 27 offsets at 90 % fill, where k_conv_pipe fetched the weights of 22 to 25 offsets
// for a third of the rows each.
//
//   step     (offset, 32 input planes): the rows and the weight slab travel with 16-byte cp.async into one of two stages
//            while the other is multiplied
//   compute  per four planes TM + TN 128-bit loads for 4 TM TN multiply-adds (16 for 256 at 128 x 64)
//
// Bound by the FMA pipe on large levels.  On levels with few tiles the offsets are divided over CTAs whose partial
// sums are added in a fixed order.  Small levels are not packed (order null, ROWS = 32): the CTA finds its offsets by
// reading its rows' column of the table.
#include <stdlib.h>

#include <algorithm>
#include <atomic>

#include "metadata.cuh"
#include "tc_ptx.cuh"

namespace scn {

int sum_partial_tiles(const float *partial, int n_split, long long n_pos, int cout, const int *order, long long n_out,
                      const float *bias, const float *bn_scale, const float *bn_shift, float leak, float *out,
                      cudaStream_t stream, unsigned char *out_split = nullptr, int out_sp = 1, int parts = 1);

namespace {

constexpr int kThreads = 128;
constexpr int kChunk = 32;            // input planes per step
constexpr int kAStride = kChunk + 4;  // four rows of a warp's broadcast loads fall on different bank quads

struct FmaParams {
  const float *in;
  long long n_in;
  float *out;  // n_split == 1: [n_out][cout]; else partial sums [n_split][positions][cout]
  long long n_out;
  const float *weight;
  const float *bias, *bn_scale, *bn_shift;
  float leak;
  const int *nbr;
  const int *order, *packed, *by_work;  // null: rows in their own order
  const unsigned *tile_bits;
  int words, K, cin, cout, n_split;
  long long n_pos;
  int *flags;
};

template <int ROWS, int BN>
struct FmaShape {
  static constexpr int TN = ROWS == 128 && BN == 64 ? 8 : 4;
  static constexpr int TX = BN / TN, TY = kThreads / TX;  // threads across planes and rows
  static constexpr int TM = ROWS / TY;
  static constexpr int STAGE = ROWS * kAStride + kChunk * BN;
  static constexpr size_t SMEM = sizeof(float) * 2 * STAGE;
  static_assert(TM >= 1 && TM * TY == ROWS, "");
};

template <int ROWS, int BN>
__global__ void __launch_bounds__(kThreads, ROWS == 128 && BN == 64 ? 3 : 4)
k_conv_fma(FmaParams P) {
  SCN_GRID_WAIT();
  using S = FmaShape<ROWS, BN>;
  constexpr int TM = S::TM, TN = S::TN;
  extern __shared__ __align__(16) float fma_smem[];
  __shared__ unsigned mask[4];
  const int tid = threadIdx.x, lane = tid & 31;
  const int tx = tid % S::TX, ty = tid / S::TX;
  // the tiles with the most offsets first (packed tiles come in ascending order of their masks)
  const long long pos0 = (P.by_work ? (long long)__ldg(P.by_work + blockIdx.x) : (long long)(gridDim.x - 1 - blockIdx.x)) * ROWS;
  const int n0 = blockIdx.y * BN;

  // ---- copying role: eight threads per row, 16 rows (of ROWS) at a time ----------------------------------------------
  const int cj = (tid & 7) * 4, cr = tid >> 3;
  constexpr int CI = ROWS / 16;

  // ---- offsets with a rule for any of the rows ------------------------------------------------------------------------
  unsigned m[4];
  if (P.order) {
    const long long t = pos0 / kOrderTile;
#pragma unroll
    for (int w = 0; w < 4; ++w) m[w] = w < P.words ? __ldg(P.tile_bits + t * P.words + w) : 0u;
  } else {
    if (tid < 4) mask[tid] = 0;
    __syncthreads();
    const long long r = pos0 + lane;  // (ROWS is 32 here)
    for (int k = tid >> 5; k < P.K; k += 4) {
      const bool hit = r < P.n_out && __ldg(P.nbr + (long long)k * P.n_out + r) >= 0;
      if (__any_sync(0xffffffffu, hit) && lane == 0) atomicOr(&mask[k >> 5], 1u << (k & 31));
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 4; ++w) m[w] = mask[w];
  }
  int n_offsets = __popc(m[0]) + __popc(m[1]) + __popc(m[2]) + __popc(m[3]);
  int skip = 0;
  if (P.n_split > 1) {  // this CTA's share of them
    skip = n_offsets * (int)blockIdx.z / P.n_split;
    n_offsets = n_offsets * ((int)blockIdx.z + 1) / P.n_split - skip;
  }
  auto next_offset = [&]() -> int {  // takes the lowest offset out of the mask
#pragma unroll
    for (int w = 0; w < 4; ++w)
      if (m[w]) {
        const int k = w * 32 + __ffs(m[w]) - 1;
        m[w] &= m[w] - 1;
        return k;
      }
    return 0;
  };
  for (int i = 0; i < skip; ++i) next_offset();
  // packed: the entries of the tile's next offset, then those of the one after, ...
  const int *packed = P.order ? P.packed + (pos0 / kOrderTile * P.K + skip) * kOrderTile + pos0 % kOrderTile + cr : nullptr;

  const int nch = (P.cin + kChunk - 1) / kChunk;
  const int steps = n_offsets * nch;
  int k_issue = 0, c_issue = 0, left = n_offsets;  // of the step to be issued next
  int v[CI];                                       // its rows' rulebook entries
  auto take_offset = [&] {
    if (left-- <= 0) return;
    k_issue = next_offset();
#pragma unroll
    for (int i = 0; i < CI; ++i) {
      if (P.order) {
        v[i] = __ldg(packed + 16 * i);
      } else {
        const long long p = pos0 + cr + 16 * i;
        v[i] = p < P.n_out ? __ldg(P.nbr + (long long)k_issue * P.n_out + p) : -1;
      }
    }
    if (P.order) packed += kOrderTile;
  };
  take_offset();
  constexpr int WP = BN / 4, WR = kThreads / WP;  // 16-byte pieces of a weight row; rows per pass
  const int wc = (tid % WP) * 4, wr = tid / WP;
  auto issue = [&](int s) {  // one cp.async group per call, empty past the end
    if (s < steps) {
      float *a = fma_smem + (s & 1) * S::STAGE, *w = a + ROWS * kAStride;
      const int c0 = c_issue * kChunk;
      if (c0 + cj < P.cin) {
        const float *src = P.in + c0 + cj;
#pragma unroll
        for (int i = 0; i < CI; ++i) {
          const bool hit = (unsigned)v[i] < (unsigned)P.n_in;
          if (v[i] >= 0 && !hit) atomicOr(P.flags, FLAG_BAD_ROW);
          cp_async16(smem_u32(a + (cr + 16 * i) * kAStride + cj), hit ? src + (long long)v[i] * P.cin : P.in, hit ? 16u : 0u);
        }
      }
      const float *wk = P.weight + ((long long)k_issue * P.cin + c0) * P.cout + n0 + wc;
      const int rows = min(kChunk, P.cin - c0);
#pragma unroll
      for (int i = 0; i < kChunk / WR; ++i) {
        const int r = wr + i * WR;
        const bool ok = r < rows && n0 + wc < P.cout;
        cp_async16(smem_u32(w + r * BN + wc), ok ? wk + (long long)r * P.cout : P.weight, ok ? 16u : 0u);
      }
      if (++c_issue == nch) {
        c_issue = 0;
        take_offset();
      }
    }
    cp_async_commit();
  };

  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int e = 0; e < TN; ++e) acc[i][e] = 0.f;

  issue(0);
  issue(1);
  int c = 0;
  for (int s = 0; s < steps; ++s) {
    cp_async_wait<1>();
    __syncthreads();
    const float *a = fma_smem + (s & 1) * S::STAGE + ty * kAStride, *w = fma_smem + (s & 1) * S::STAGE + ROWS * kAStride + tx * 4;
    const int kmax = min(kChunk, P.cin - c * kChunk);
    auto four = [&](int kk) {
      float4 wv[4][TN / 4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int h = 0; h < TN / 4; ++h) wv[q][h] = *reinterpret_cast<const float4 *>(w + (kk + q) * BN + h * (BN / 2));
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float4 av = *reinterpret_cast<const float4 *>(a + i * S::TY * kAStride + kk);
        const float ax[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int h = 0; h < TN / 4; ++h) {
            float *o = &acc[i][h * 4];
            o[0] = fmaf(ax[q], wv[q][h].x, o[0]);
            o[1] = fmaf(ax[q], wv[q][h].y, o[1]);
            o[2] = fmaf(ax[q], wv[q][h].z, o[2]);
            o[3] = fmaf(ax[q], wv[q][h].w, o[3]);
          }
      }
    };
    if (kmax == kChunk) {
#pragma unroll 2
      for (int kk = 0; kk < kChunk; kk += 4) four(kk);
    } else {
      for (int kk = 0; kk < kmax; kk += 4) four(kk);
    }
    if (++c == nch) c = 0;
    __syncthreads();
    issue(s + 2);
  }

  // ---- each row's planes, written once ------------------------------------------------------------------------------
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const long long p = pos0 + ty + i * S::TY;
    const int r = P.order ? __ldg(P.order + p) : p < P.n_out ? (int)p : -1;
    if (r < 0) continue;
#pragma unroll
    for (int h = 0; h < TN / 4; ++h) {
      const int n = n0 + tx * 4 + h * (BN / 2);
      if (n >= P.cout) continue;
      float4 q = make_float4(acc[i][h * 4], acc[i][h * 4 + 1], acc[i][h * 4 + 2], acc[i][h * 4 + 3]);
      if (P.n_split > 1) {
        *reinterpret_cast<float4 *>(P.out + ((long long)blockIdx.z * P.n_pos + p) * P.cout + n) = q;
        continue;
      }
      if (P.bias) {
        const float4 b = __ldg(reinterpret_cast<const float4 *>(P.bias + n));
        q.x += b.x, q.y += b.y, q.z += b.z, q.w += b.w;
      }
      if (P.bn_scale) {  // separate multiply and add, as the stand-alone BatchNorm kernel rounds them
        const float4 sc = __ldg(reinterpret_cast<const float4 *>(P.bn_scale + n)), sh = __ldg(reinterpret_cast<const float4 *>(P.bn_shift + n));
        q.x = __fadd_rn(__fmul_rn(q.x, sc.x), sh.x), q.y = __fadd_rn(__fmul_rn(q.y, sc.y), sh.y);
        q.z = __fadd_rn(__fmul_rn(q.z, sc.z), sh.z), q.w = __fadd_rn(__fmul_rn(q.w, sc.w), sh.w);
        q.x *= q.x > 0.f ? 1.f : P.leak, q.y *= q.y > 0.f ? 1.f : P.leak;
        q.z *= q.z > 0.f ? 1.f : P.leak, q.w *= q.w > 0.f ? 1.f : P.leak;
      }
      *reinterpret_cast<float4 *>(P.out + (long long)r * P.cout + n) = q;
    }
  }
}

template <int ROWS, int BN>
int launch_fma(const FmaParams &P, cudaStream_t stream) {
  using S = FmaShape<ROWS, BN>;
  static std::atomic<bool> configured[64];
  int dev = 0;
  SCN_CUDA_CHECK(cudaGetDevice(&dev));
  SCN_REQUIRE(dev >= 0 && dev < 64, SCN_ERR_UNSUPPORTED, "device index %d unsupported", dev);
  if (!configured[dev].load()) {
    SCN_CUDA_CHECK(cudaFuncSetAttribute(k_conv_fma<ROWS, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM));
    configured[dev].store(true);
  }
  auto kernel = k_conv_fma<ROWS, BN>;
  SCN_LAUNCH(kernel, dim3((unsigned)(P.n_pos / ROWS), (unsigned)ceil_div(P.cout, BN), (unsigned)P.n_split), kThreads, S::SMEM, stream, P);
  SCN_CUDA_CHECK(cudaGetLastError());
  return SCN_OK;
}

}  // namespace

bool conv_fma_supported(const float *in, const float *out, const float *weight, const float *bias, int K, int cin, int cout,
                        int groups) {
  return groups == 1 && K <= kOrderMaxOffsets && cin % 4 == 0 && cout % 4 == 0 &&
         ((uintptr_t)in | (uintptr_t)out | (uintptr_t)weight | (uintptr_t)bias) % 16 == 0;
}

// Below this many rows the rows are not packed: a layer takes about as long as the packing's launch.
bool conv_fma_wants_order(long long n_out) { return n_out >= 2048; }

// out [n_out, cout] = act((bias + sum_k in[table[k][.]] @ W[k]) * bn_scale + bn_shift); `ord` null: unpacked rows
int conv_forward_fma(const float *in, long long n_in, float *out, long long n_out, const float *weight, const float *bias,
                     const float *bn_scale, const float *bn_shift, float leak, const int *table, const RowOrder *ord, int K,
                     int cin, int cout, int *flags, cudaStream_t stream) {
  if (n_out == 0) return SCN_OK;
  FmaParams P{};
  P.in = in;
  P.n_in = n_in;
  P.out = out;
  P.n_out = n_out;
  P.weight = weight;
  P.bias = bias;
  P.bn_scale = bn_scale;
  P.bn_shift = bn_shift;
  P.leak = leak;
  P.nbr = table;
  P.order = ord ? ord->order : nullptr;
  P.packed = ord ? ord->packed : nullptr;
  P.by_work = ord ? ord->by_work : nullptr;  // (tiles are ROWS = 128 rows then)
  P.tile_bits = ord ? ord->tile_bits : nullptr;
  P.words = ord ? ord->words : 0;
  P.K = K;
  P.cin = cin;
  P.cout = cout;
  P.flags = flags;
  // 64 planes per CTA unless that leaves half of them unused; 128 rows where they are packed (16 shared-memory loads for
  // 256 multiply-adds instead of 8 for 64), 32 otherwise; then the offsets over as many CTAs as still leave each about
  // four steps
  const int bn = cout <= 16 ? 16 : cout <= 32 || (cout % 64 != 0 && cout % 64 <= 32 && cout < 128) ? 32 : 64;
  const long long cols = ceil_div(cout, bn);
  const int rows = ord ? 128 : 32;
  P.n_pos = ord ? ord->n_tiles * kOrderTile : ceil_div(n_out, 32) * 32;
  const long long ctas = P.n_pos / rows * cols;
  const int offsets = ord && ord->one_offset ? 1 : K;  // of a tile
  const int steps = (int)(offsets * ceil_div(cin, kChunk));
  P.n_split = (int)std::max<long long>(1, std::min<long long>({ceil_div(148 * 3, ctas), (long long)steps / 4, (long long)offsets, 16ll}));
  if (const char *e = getenv("SCN_FMA_SPLIT")) P.n_split = std::max(1, std::min(atoi(e), 64));
  float *partial = nullptr;
  if (P.n_split > 1) {
    SCN_TRY(device_alloc((void **)&partial, sizeof(float) * (size_t)P.n_split * P.n_pos * cout, stream));
    P.out = partial;
  }
  int rc;
  if (rows == 128)
    rc = bn == 64 ? launch_fma<128, 64>(P, stream) : bn == 32 ? launch_fma<128, 32>(P, stream) : launch_fma<128, 16>(P, stream);
  else
    rc = bn == 64 ? launch_fma<32, 64>(P, stream) : bn == 32 ? launch_fma<32, 32>(P, stream) : launch_fma<32, 16>(P, stream);
  if (rc == SCN_OK && P.n_split > 1)
    rc = sum_partial_tiles(partial, P.n_split, P.n_pos, cout, P.order, n_out, bias, bn_scale, bn_shift, leak, out, stream);
  device_free(partial, stream);
  return rc;
}

}  // namespace scn
