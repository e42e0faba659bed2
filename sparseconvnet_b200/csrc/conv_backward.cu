// Backward pass of the three convolution operators (the reference: CPU/Convolution.cpp:80-115,
// 152-190, CPU/Deconvolution.cpp, CUDA/Convolution.cu dConvolution_KMxKN_backward_dW*), fp32.
//
//   d_input   the same output-stationary kernels as the forward pass, run on the opposite table
//             of the dense rulebook with the weights transposed per offset:
//                 d_in[i] = sum_k d_out[t[k][i]] * W[k]^T
//             (t = tnbr for SubmanifoldConvolution / Convolution, nbr for Deconvolution);
//   d_weight  d_W[k] = sum over the rules (i, o) of offset k of in[i]^T d_out[o]: the rules are cut
//             into chunks of rulebook entries, every CTA reduces one chunk of one offset into a
//             32 x 32 tile, and the chunks' partial tiles are added in a fixed order, so the
//             result is bit-reproducible (no floating-point atomics);
//   d_bias    column sums of d_out, the same two steps.
#include <algorithm>

#include <stdlib.h>

#include <atomic>

#include "metadata.cuh"
#include "tc_ptx.cuh"

namespace scn {

extern std::atomic<int> g_backward_precision;
int conv_forward_table(Rulebook &rb, bool transposed_table, const float *in, long long rows_in, float *out,
                       long long rows_out, const float *weight, const float *bias, int cin, int cout, int groups,
                       int precision, int *flags, cudaStream_t stream, const float *bn_scale = nullptr,
                       const float *bn_shift = nullptr, float leak = 1.f, const float *pre_scale = nullptr,
                       const float *pre_shift = nullptr, float pre_leak = 1.f, const float *in_b = nullptr,
                       int planes_a = 0);
int conv_forward_simt(const float *in, long long n_in, float *out, long long n_out, const float *weight,
                      const float *bias, const int *table, int K, int cin, int cout, int groups, int *flags,
                      cudaStream_t stream);

bool dweight_tile_supported(const float *in, const float *d_out, const Rulebook &rb, int cin, int cout);
int dweight_tile(const float *in, long long rows_in, const float *d_out, long long rows_out, const Rulebook &rb,
                 bool swap, int cin, int cout, float *d_weight, int *flags, cudaStream_t stream);

// W [K][groups][cin][cout] -> [K][groups][cout][cin]; mirror_groups > 0 (the number of groups): offset k goes to K - 1 - k
__global__ void k_transpose_weight(const float *__restrict__ w, float *__restrict__ wt, long long n_mats, int cin,
                                   int cout, int mirror_groups) {
  SCN_GRID_WAIT();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long per = (long long)cin * cout;
  if (idx >= n_mats * per) return;
  const long long m = idx / per;
  const int c = (int)((idx % per) / cout), n = (int)(idx % cout);
  const long long to = mirror_groups ? n_mats - (m / mirror_groups + 1) * mirror_groups + m % mirror_groups : m;
  wt[to * per + (long long)n * cin + c] = w[idx];
}

// partial[chunk][k][g][c][n] = sum over the chunk's rulebook entries j of offset k of
//   in[in_row(j)][g*cin + c] * d_out[out_row(j)][g*cout + n]
// where (in_row, out_row) = (nbr[k][j], j), or (j, nbr[k][j]) when the operator runs the rulebook
// backwards (Deconvolution); nbr null: (j, j), a dense product.  grid = (chunks, K, groups * c-tiles * n-tiles), 256 threads,
// 32 x 32 tile, 2 x 2 outputs per thread.
__global__ void __launch_bounds__(256)
k_conv_dweight(const float *__restrict__ in, int ld_in, long long n_in_rows, const float *__restrict__ dout,
               int ld_out, long long n_out_rows, const int *__restrict__ nbr, long long n_entries, int swap,
               int cin, int cout, int groups, long long chunk_rows, float *__restrict__ partial, int *flags) {
  SCN_GRID_WAIT();
  __shared__ float A[32][33], B[32][33];
  const int tid = threadIdx.x;
  const int k = blockIdx.y;
  const int tiles_c = (cin + 31) / 32, tiles_n = (cout + 31) / 32;
  int z = blockIdx.z;
  const int tn = z % tiles_n;
  z /= tiles_n;
  const int tc = z % tiles_c;
  const int g = z / tiles_c;
  const int c0 = tc * 32, n0 = tn * 32;
  const long long j0 = (long long)blockIdx.x * chunk_rows;
  const long long j1 = min(n_entries, j0 + chunk_rows);
  const int lr = tid >> 3, lq = (tid & 7) * 4;  // loader: row of the 32-entry slab, first of 4 columns
  const int ty = tid >> 4, tx = tid & 15;       // 2 x 2 outputs at (2 ty, 2 tx)
  float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
  for (long long jb = j0; jb < j1; jb += 32) {
    const long long j = jb + lr;
    long long ri = -1, ro = -1;
    if (j < j1) {
      const int a = nbr ? nbr[(long long)k * n_entries + j] : (int)j;
      if (a >= 0) {
        ri = swap ? j : a;
        ro = swap ? a : j;
        if (ri >= n_in_rows || ro >= n_out_rows) {
          atomicOr(flags, FLAG_BAD_ROW);
          ri = ro = -1;
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int c = c0 + lq + e, n = n0 + lq + e;
      A[lr][lq + e] = (ri >= 0 && c < cin) ? in[ri * ld_in + g * cin + c] : 0.f;
      B[lr][lq + e] = (ro >= 0 && n < cout) ? dout[ro * ld_out + g * cout + n] : 0.f;
    }
    __syncthreads();
#pragma unroll 8
    for (int r = 0; r < 32; ++r) {
      const float a0 = A[r][2 * ty], a1 = A[r][2 * ty + 1], b0 = B[r][2 * tx], b1 = B[r][2 * tx + 1];
      acc[0][0] = fmaf(a0, b0, acc[0][0]);
      acc[0][1] = fmaf(a0, b1, acc[0][1]);
      acc[1][0] = fmaf(a1, b0, acc[1][0]);
      acc[1][1] = fmaf(a1, b1, acc[1][1]);
    }
    __syncthreads();
  }
  float *dst = partial + (((long long)blockIdx.x * gridDim.y + k) * groups + g) * cin * cout;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int jn = 0; jn < 2; ++jn) {
      const int c = c0 + 2 * ty + i, n = n0 + 2 * tx + jn;
      if (c < cin && n < cout) dst[(long long)c * cout + n] = acc[i][jn];
    }
}

// out[i] = sum over chunks, in order, of partial[chunk][i]; `add`: behind what is there already
__global__ void k_sum_chunks(const float *__restrict__ partial, int chunks, long long n, float *__restrict__ out, bool add) {
  SCN_GRID_WAIT();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float acc = add ? out[i] : 0.f;
  int c = 0;
  for (; c + 8 <= chunks; c += 8) {  // eight loads on their way
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = partial[(long long)(c + u) * n + i];
#pragma unroll
    for (int u = 0; u < 8; ++u) acc += v[u];
  }
  for (; c < chunks; ++c) acc += partial[(long long)c * n + i];
  out[i] = acc;
}

// The same partial sums on the warp-level tensor path (groups = 1, any plane counts): a CTA owns one offset, one chunk
// of its rulebook column and a tile of 32 WM x 32 WN weights.  It keeps only the entries that hold a rule (a third of
// them on surface data), in a list in shared memory, and walks the list in steps of 32 or 64 rules: the rules' input and
// output rows travel with cp.async through a ring of stages, then each warp multiplies
// in^T [32 x 8 rules] x d_out [8 rules x 32] per block of eight rules with mma.sync.m16n8k8 on the hi/lo split of both
// operands (hi x hi + hi x lo + lo x hi; as accurate as fp32 multiply-adds, see dw_split and the sums).  With few 32 x 32 tiles several warps
// share the blocks of a step and their sums are added in warp order, so the result does not depend on timing.  Plane
// counts that are no multiple of the tile are padded with zeros in the stage only.
//
// Bound by the tensor instructions (three passes of tf32: 92 TFLOP/s).  Reading every fragment value of every rule
// straight from the matrices, once per 32 x 32 tile, was bound by the loads.
__device__ __forceinline__ void dw_mma(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// x = hi + lo, both rounded to the nearest tf32: what is left out (lo x lo and a bit of lo, 2^-23 of x) has either sign as
// often as the other.  Cut off instead of rounded it all had the sign of x: 8e-6 of a sum of 100 k products of one sign, 1e-7
// now, and 4e-6 against 2e-7 with signs mixed.
__device__ __forceinline__ void dw_split(float x, unsigned &hi, unsigned &lo) {
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(x - __uint_as_float(hi)));
}
__device__ __forceinline__ void dw_copy4(unsigned dst, const float *src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(ok ? 4u : 0u) : "memory");
}

// WM x WN warps side by side, each with 16 MT x 32 weights (MT 1: layers of at most 16 input planes)
template <int WM, int WN, int MT>
struct DwShape {
  static constexpr int M = 16 * MT * WM, N = 32 * WN;
  static constexpr int SHARE = WM * WN == 1 ? 4 : WM * WN <= 3 ? 2 : 1;  // warps that share a 32 x 32 tile
  static constexpr int THREADS = 32 * WM * WN * SHARE;
  static constexpr int STEP = SHARE == 4 ? 64 : 32, STAGES = 3;
  static constexpr int LOADS = 8, LIST = LOADS * THREADS;  // entries looked at in one go
  static constexpr int SA = M + 8, SB = N + 8;  // row strides: rules t and planes g of a fragment fall on different banks
  static constexpr int STAGE = STEP * (SA + SB);
  static constexpr int TILE = 32 * 33;          // a warp's result, in the stages' memory
  static constexpr size_t SMEM = sizeof(float) * STAGES * STAGE + sizeof(int2) * LIST;
  static_assert(STAGES * STAGE >= (THREADS / 32) * TILE, "the warps' results do not fit the stages");
};

template <int WM, int WN, int MT>
__global__ void __launch_bounds__(DwShape<WM, WN, MT>::THREADS)
k_conv_dweight_mma(const float *__restrict__ in, int ld_in, long long n_in_rows, const float *__restrict__ dout,
                   int ld_out, long long n_out_rows, const int *__restrict__ nbr, long long n_entries, int swap,
                   int cin, int cout, int vec_in, int vec_out, long long chunk_rows, float *__restrict__ partial, int *flags) {
  SCN_GRID_WAIT();
  using S = DwShape<WM, WN, MT>;
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int kWarps = S::THREADS / 32;
  extern __shared__ __align__(16) unsigned char dw_smem[];
  float *stages = reinterpret_cast<float *>(dw_smem);
  int2 *list = reinterpret_cast<int2 *>(stages + S::STAGES * S::STAGE);
  __shared__ int counts[S::LOADS][kWarps];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int k = blockIdx.y;
  const int tiles_n = (cout + S::N - 1) / S::N;
  const int c0 = ((int)blockIdx.z / tiles_n) * S::M, n0 = ((int)blockIdx.z % tiles_n) * S::N;
  const int mw = warp % WM, nw = (warp / WM) % WN, share = warp / (WM * WN);
  const long long j0 = (long long)blockIdx.x * chunk_rows, j1 = min(n_entries, j0 + chunk_rows);
  const int *col = nbr + (long long)k * n_entries;
  // planes of the tile that exist; rows that are copied value by value leave the others the zeros they start as
  const int cols_in = min(S::M, cin - c0), cols_out = min(S::N, cout - n0);
  if (!vec_in || !vec_out) {
    for (int i = tid; i < S::STAGES * S::STAGE; i += S::THREADS) stages[i] = 0.f;
    __syncthreads();
  }

  // The tensor core cuts off what does not fit its running sum, always towards zero: it adds up eight rules at a time
  // (from zero), and fp32 additions add those.
  float d[MT][4][4];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) d[mt][nt][0] = d[mt][nt][1] = d[mt][nt][2] = d[mt][nt][3] = 0.f;

  // the rows of step `s` of a list of `n` rules into stage `s % STAGES`; one cp.async group per call
  auto issue = [&](int s, int n) {
    float *a = stages + (s % S::STAGES) * S::STAGE, *b = a + S::STEP * S::SA;
    if (s * S::STEP < n) {
      if (vec_in) {
#pragma unroll 4
        for (int i = tid; i < S::STEP * (S::M / 4); i += S::THREADS) {
          const int r = i / (S::M / 4), c = (i % (S::M / 4)) * 4, e = s * S::STEP + r;
          const bool ok = e < n && c < cols_in;
          cp_async16(smem_u32(a + r * S::SA + c), ok ? in + (long long)list[e].x * ld_in + c0 + c : in, ok ? 16u : 0u);
        }
      } else {
        for (int i = tid; i < S::STEP * cols_in; i += S::THREADS) {
          const int r = i / cols_in, c = i - r * cols_in, e = s * S::STEP + r;
          dw_copy4(smem_u32(a + r * S::SA + c), e < n ? in + (long long)list[e].x * ld_in + c0 + c : in, e < n);
        }
      }
      if (vec_out) {
#pragma unroll 4
        for (int i = tid; i < S::STEP * (S::N / 4); i += S::THREADS) {
          const int r = i / (S::N / 4), c = (i % (S::N / 4)) * 4, e = s * S::STEP + r;
          const bool ok = e < n && c < cols_out;
          cp_async16(smem_u32(b + r * S::SB + c), ok ? dout + (long long)list[e].y * ld_out + n0 + c : dout, ok ? 16u : 0u);
        }
      } else {
        for (int i = tid; i < S::STEP * cols_out; i += S::THREADS) {
          const int r = i / cols_out, c = i - r * cols_out, e = s * S::STEP + r;
          dw_copy4(smem_u32(b + r * S::SB + c), e < n ? dout + (long long)list[e].y * ld_out + n0 + c : dout, e < n);
        }
      }
    }
    cp_async_commit();
  };

  for (long long jb = j0; jb < j1; jb += S::LIST) {
    // ---- the rules among the next LIST entries, in entry order -----------------------------------------------------
    int v[S::LOADS];
    unsigned m[S::LOADS];
#pragma unroll
    for (int u = 0; u < S::LOADS; ++u) {
      const long long j = jb + u * S::THREADS + tid;
      v[u] = j < j1 ? __ldg(col + j) : -1;
    }
#pragma unroll
    for (int u = 0; u < S::LOADS; ++u) {
      if (v[u] >= (swap ? n_out_rows : n_in_rows)) {
        atomicOr(flags, FLAG_BAD_ROW);
        v[u] = -1;
      }
      m[u] = __ballot_sync(kFull, v[u] >= 0);
      if (lane == 0) counts[u][warp] = __popc(m[u]);
    }
    __syncthreads();
    int n = 0;
#pragma unroll
    for (int u = 0; u < S::LOADS; ++u) {
      int at = n;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        if (w < warp) at += counts[u][w];
        n += counts[u][w];
      }
      const int j = (int)(jb + u * S::THREADS + tid);
      if (v[u] >= 0) list[at + __popc(m[u] & ((1u << lane) - 1u))] = swap ? make_int2(j, v[u]) : make_int2(v[u], j);
    }
    __syncthreads();
    // ---- the list in steps -------------------------------------------------------------------------------------------
    const int steps = (n + S::STEP - 1) / S::STEP;
#pragma unroll
    for (int s = 0; s < S::STAGES - 1; ++s) issue(s, n);
    for (int s = 0; s < steps; ++s) {
      cp_async_wait<S::STAGES - 2>();
      __syncthreads();  // the step has landed for everybody, and the step before is consumed
      issue(s + S::STAGES - 1, n);
      const float *a = stages + (s % S::STAGES) * S::STAGE + mw * 16 * MT, *b = stages + (s % S::STAGES) * S::STAGE + S::STEP * S::SA + nw * 32;
#pragma unroll
      for (int kb = 0; kb < S::STEP / 8 / S::SHARE; ++kb) {
        const int r0 = (kb * S::SHARE + share) * 8 + t;
        const float *a0 = a + r0 * S::SA + g, *a1 = a0 + 4 * S::SA, *b0 = b + r0 * S::SB + g, *b1 = b0 + 4 * S::SB;
        unsigned ah[MT][4], al[MT][4], bh[4][2], bl[4][2];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {  // A[m = plane][k = rule]: a0 (g, t), a1 (g + 8, t), a2 (g, t + 4), a3 (g + 8, t + 4)
          dw_split(a0[mt * 16], ah[mt][0], al[mt][0]);
          dw_split(a0[mt * 16 + 8], ah[mt][1], al[mt][1]);
          dw_split(a1[mt * 16], ah[mt][2], al[mt][2]);
          dw_split(a1[mt * 16 + 8], ah[mt][3], al[mt][3]);
        }
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {  // B[k = rule][n = plane]: b0 (t, g), b1 (t + 4, g)
          dw_split(b0[nt * 8], bh[nt][0], bl[nt][0]);
          dw_split(b1[nt * 8], bh[nt][1], bl[nt][1]);
        }
        float p[MT][4][4] = {};
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) dw_mma(p[mt][nt], al[mt], bh[nt]);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) dw_mma(p[mt][nt], ah[mt], bl[nt]);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) dw_mma(p[mt][nt], ah[mt], bh[nt]);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) d[mt][nt][e] += p[mt][nt][e];
      }
    }
    cp_async_wait<0>();
    __syncthreads();
  }

  // ---- the warps' tiles; those of warps that shared one are added in warp order ------------------------------------
  float *tile = stages + warp * S::TILE;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {  // d0 (g, 2t), d1 (g, 2t + 1), d2 (g + 8, 2t), d3 (g + 8, 2t + 1)
      float *q = tile + (mt * 16 + g) * 33 + nt * 8 + 2 * t;
      q[0] = d[mt][nt][0];
      q[1] = d[mt][nt][1];
      q[8 * 33] = d[mt][nt][2];
      q[8 * 33 + 1] = d[mt][nt][3];
    }
  __syncthreads();
  float *dst = partial + ((long long)blockIdx.x * gridDim.y + k) * cin * cout;
  for (int i = tid; i < S::M * S::N; i += S::THREADS) {
    const int c = i / S::N, n = i % S::N;
    if (c0 + c >= cin || n0 + n >= cout) continue;
    const float *q = stages + (c / (16 * MT) + (n / 32) * WM) * S::TILE + c % (16 * MT) * 33 + n % 32;  // share 0 of the tile
    float v = q[0];
#pragma unroll
    for (int w = 1; w < S::SHARE; ++w) v += q[w * WM * WN * S::TILE];
    dst[(long long)(c0 + c) * cout + n0 + n] = v;
  }
}

static int n_chunks(long long rows) { return (int)std::max<long long>(1, std::min<long long>(64, rows / 4096)); }

template <int WM, int WN, int MT = 2>
static int launch_dweight(const float *in, int ld_in, long long n_in_rows, const float *dout, int ld_out,
                          long long n_out_rows, const int *nbr, long long n_entries, int swap, int K, int cin, int cout,
                          float *d_weight, int *flags, cudaStream_t stream) {
  using S = DwShape<WM, WN, MT>;
  static std::atomic<bool> configured[64];
  int dev = 0;
  SCN_CUDA_CHECK(cudaGetDevice(&dev));
  SCN_REQUIRE(dev >= 0 && dev < 64, SCN_ERR_UNSUPPORTED, "device index %d unsupported", dev);
  SCN_REQUIRE(n_entries < (1ll << 31), SCN_ERR_UNSUPPORTED, "%lld rulebook entries", n_entries);
  if (!configured[dev].load()) {
    SCN_CUDA_CHECK(cudaFuncSetAttribute(k_conv_dweight_mma<WM, WN, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM));
    configured[dev].store(true);
  }
  // about four waves of the CTAs the SMs hold, in chunks of whole lists; no fewer than one per 4096 entries (up to 64), which
  // bounds how many additions a sum goes through before the chunks' sums are added
  const int tiles = (int)(ceil_div(cin, S::M) * ceil_div(cout, S::N));
  const int per_sm = std::max(1, (int)(220 * 1024 / S::SMEM));
  const long long wanted = std::max<long long>(ceil_div(148 * 4 * per_sm, (long long)K * tiles), n_chunks(n_entries));
  const int chunks = (int)std::max<long long>(1, std::min<long long>(wanted, n_entries / S::LIST));
  const long long chunk_rows = ceil_div(ceil_div(n_entries, chunks), S::LIST) * S::LIST;
  const int grid_x = (int)ceil_div(n_entries, chunk_rows);
  const long long w_elems = (long long)K * cin * cout;
  Scratch tmp(stream);
  float *partial = d_weight;
  if (grid_x > 1) SCN_TRY(tmp.get(&partial, sizeof(float) * (size_t)grid_x * w_elems));
  const int vec_in = cin % 4 == 0 && ld_in % 4 == 0 && (uintptr_t)in % 16 == 0;
  const int vec_out = cout % 4 == 0 && ld_out % 4 == 0 && (uintptr_t)dout % 16 == 0;
  SCN_LAUNCH((k_conv_dweight_mma<WM, WN, MT>), dim3((unsigned)grid_x, (unsigned)K, (unsigned)tiles), S::THREADS, S::SMEM, stream, in, ld_in, n_in_rows, dout, ld_out, n_out_rows, nbr, n_entries, swap, cin, cout, vec_in, vec_out, chunk_rows, partial, flags);
  if (grid_x > 1)
    SCN_LAUNCH(k_sum_chunks, (unsigned)ceil_div(w_elems, 256), 256, 0, stream, partial, grid_x, w_elems, d_weight, false);
  SCN_CUDA_CHECK(cudaGetLastError());
  return SCN_OK;
}

// Up to three input planes (the first layer of a network) and 32 output planes: no matrix to speak of.  A lane owns an
// output plane and keeps the sums of nine offsets x CIN planes in registers, in full fp32; d_out rows are read as they lie.
// Per batch of 32 rows a warp fetches the nine table entries of a row and the inputs they name with one lane per row, leaves
// them in shared memory (zeros where there is no rule) and reads them back row by row, the same for all lanes.  Most
// multiply-adds of surface data are with such zeros, which is cheaper than finding the others; bound by the L1 pipe (the
// scattered 4-byte loads, and the shared memory both ways).  k_conv_dweight_mma, whose steps are padded to 16 planes, took
// 218 us for 3 -> 32 planes of two rooms (120 now), 28 for 3 k rows (8), 41 for 1 -> 16 planes on 100 k pixels (15); with four
// input planes (97 against 120 us at 400 k scattered rows) and with two blocks of output planes (141, 184) it stays ahead.
constexpr int kThinOffsets = 9;

template <int CIN>
__global__ void __launch_bounds__(256, 2)
k_conv_dweight_thin(const float *__restrict__ in, long long n_in, const float *__restrict__ dout, long long n_out,
                    const int *__restrict__ nbr, int K, int cout, long long chunk_rows, float *__restrict__ partial, int *flags) {
  SCN_GRID_WAIT();
  constexpr int N = kThinOffsets * CIN, W = (N + 3) / 4 * 4;  // values of a row
  __shared__ __align__(16) float values[8][32][W];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int blocks_p = (cout + 31) / 32, k0 = (int)blockIdx.y / blocks_p * kThinOffsets, p = (int)blockIdx.y % blocks_p * 32 + lane;
  const int n_off = min(kThinOffsets, K - k0);
  const long long begin = blockIdx.x * chunk_rows, end = min(n_out, begin + chunk_rows);
  float acc[N];
#pragma unroll
  for (int i = 0; i < N; ++i) acc[i] = 0.f;
  bool bad = false;
  int e[kThinOffsets];
  auto fetch = [&](long long row) {
#pragma unroll
    for (int k = 0; k < kThinOffsets; ++k) e[k] = k < n_off && row < end ? __ldg(nbr + (long long)(k0 + k) * n_out + row) : -1;
  };
  fetch(begin + warp * 32 + lane);
  for (long long r0 = begin + warp * 32; r0 < end; r0 += 256) {
#pragma unroll
    for (int k = 0; k < kThinOffsets; ++k) {
      const bool hit = (unsigned)e[k] < (unsigned long long)n_in;
      bad |= e[k] >= n_in;
#pragma unroll
      for (int c = 0; c < CIN; ++c) values[warp][lane][k * CIN + c] = hit ? __ldg(in + (long long)e[k] * CIN + c) : 0.f;
    }
    fetch(r0 + 256 + lane);  // the next batch's, on their way while this one is summed
    __syncwarp();
    const int rows = (int)min(32ll, end - r0);
    for (int r = 0; r < rows; r += 8) {
      float d[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) d[u] = r + u < rows && p < cout ? __ldg(dout + (r0 + r + u) * cout + p) : 0.f;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float4 *v = reinterpret_cast<const float4 *>(values[warp][r + u]);
#pragma unroll
        for (int i = 0; i < W / 4; ++i) {
          const float4 x = v[i];
          acc[i * 4] = fmaf(x.x, d[u], acc[i * 4]);
          if (i * 4 + 1 < N) acc[i * 4 + 1] = fmaf(x.y, d[u], acc[i * 4 + 1]);
          if (i * 4 + 2 < N) acc[i * 4 + 2] = fmaf(x.z, d[u], acc[i * 4 + 2]);
          if (i * 4 + 3 < N) acc[i * 4 + 3] = fmaf(x.w, d[u], acc[i * 4 + 3]);
        }
      }
    }
    __syncwarp();
  }
  if (bad) atomicOr(flags, FLAG_BAD_ROW);
  // the warps' sums in order
  __syncthreads();
  float(*sums)[N][32] = reinterpret_cast<float(*)[N][32]>(&values[0][0][0]);
#pragma unroll
  for (int i = 0; i < N; ++i) sums[warp][i][lane] = acc[i];
  __syncthreads();
  if (p >= cout) return;
  for (int i = warp; i < n_off * CIN; i += 8) {
    float x = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) x += sums[w][i][lane];
    partial[(((long long)blockIdx.x * K + k0) * CIN + i) * cout + p] = x;  // [chunk][offset][input plane][output plane]
  }
}

static int dweight_thin(const float *in, long long rows_in, const float *d_out, long long rows_out, const int *nbr, int K, int cin,
                        int cout, float *d_weight, int *flags, cudaStream_t stream) {
  // one wave of two CTAs per SM, in whole batches
  const int columns = (int)(ceil_div(K, kThinOffsets) * ceil_div(cout, 32));
  const long long wanted = std::max<long long>(1, std::min<long long>(148 * 2 / columns, ceil_div(rows_out, 256)));
  const long long chunk_rows = ceil_div(ceil_div(rows_out, wanted), 256) * 256;
  const int chunks = (int)ceil_div(rows_out, chunk_rows);
  const long long w_elems = (long long)K * cin * cout;
  Scratch tmp(stream);
  float *partial = d_weight;
  if (chunks > 1) SCN_TRY(tmp.get(&partial, sizeof(float) * (size_t)chunks * w_elems));
  const auto kernel = cin == 1 ? k_conv_dweight_thin<1> : cin == 2 ? k_conv_dweight_thin<2> : k_conv_dweight_thin<3>;
  SCN_LAUNCH(kernel, dim3((unsigned)chunks, (unsigned)columns), 256, 0, stream, in, rows_in, d_out, rows_out, nbr, K, cout, chunk_rows, partial, flags);
  if (chunks > 1)
    SCN_LAUNCH(k_sum_chunks, (unsigned)ceil_div(w_elems, 256), 256, 0, stream, partial, chunks, w_elems, d_weight, false);
  SCN_CUDA_CHECK(cudaGetLastError());
  return SCN_OK;
}

// 32-plane tiles per side: one CTA tile up to 96 planes, beyond that whichever of 64 and 96 pads less.  Few entries
// make few chunks, and tiles of 32 x 32 fill the SMs instead: 80 x 80 weights on 7 k rows 84 against 381 us, 25 k rows 191
// against 382, 96 x 48 on 25 k rows 134 against 213; from about 50 k rows on the second fetch of the rows costs as much
// (48 x 48 on 56 k rows 169 against 160 us, on 160 k rows 375 against 291).
static int dweight_side(int planes, long long n_entries) {
  if (n_entries < 32768) return 1;
  if (planes <= 96) return (planes + 31) / 32;
  return ceil_div(planes, 96) * 96 < ceil_div(planes, 64) * 64 ? 3 : 2;
}

// partial[chunk][p] = sum over the chunk's rows of x[row][p]; grid = (plane tiles of 32, chunks)
__global__ void __launch_bounds__(256)
k_column_sums(const float *__restrict__ x, long long n_rows, int planes, long long chunk_rows,
              float *__restrict__ partial) {
  SCN_GRID_WAIT();
  __shared__ float sh[8][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int p = blockIdx.x * 32 + lane;
  const long long r0 = (long long)blockIdx.y * chunk_rows, r1 = min(n_rows, r0 + chunk_rows);
  float s = 0.f;
  if (p < planes)
    for (long long r = r0 + w; r < r1; r += 8) s += x[r * planes + p];
  sh[w][lane] = s;
  __syncthreads();
  if (w == 0 && p < planes) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += sh[i][lane];
    partial[(long long)blockIdx.y * planes + p] = t;
  }
}

static std::atomic<int> g_last_dweight_kernel{-1};

// Runs the backward pass for one operator call.  `transposed` as in the forward pass (Deconvolution).
static int run_conv_backward(scn_metadata *md, Rulebook &rb, bool transposed, const float *in, float *d_in,
                             const float *d_out, const float *weight, float *d_weight, float *d_bias,
                             int n_in_planes, int n_out_planes, int groups, cudaStream_t stream) {
  SCN_REQUIRE(groups >= 1 && n_in_planes >= 1 && n_out_planes >= 1 && n_in_planes % groups == 0 &&
                  n_out_planes % groups == 0,
              SCN_ERR_BAD_ARG, "planes %d -> %d not divisible into %d groups", n_in_planes, n_out_planes, groups);
  SCN_REQUIRE(weight && d_weight, SCN_ERR_BAD_ARG, "null weight or weight gradient");
  const int cin = n_in_planes / groups, cout = n_out_planes / groups, K = rb.n_offsets;
  const long long rows_in = transposed ? rb.n_out : rb.n_in;
  const long long rows_out = transposed ? rb.n_in : rb.n_out;
  const long long w_elems = (long long)K * groups * cin * cout;
  if (!md->flags_dev) {
    SCN_TRY(device_alloc((void **)&md->flags_dev, sizeof(int), stream));
    SCN_CUDA_CHECK(cudaMemsetAsync(md->flags_dev, 0, sizeof(int), stream));
  }
  if (rows_out == 0 || rows_in == 0) {  // no rule: gradients are zero
    SCN_CUDA_CHECK(cudaMemsetAsync(d_weight, 0, sizeof(float) * (size_t)w_elems, stream));
    if (d_bias) SCN_CUDA_CHECK(cudaMemsetAsync(d_bias, 0, sizeof(float) * (size_t)n_out_planes, stream));
    if (rows_in > 0 && d_in)
      SCN_CUDA_CHECK(cudaMemsetAsync(d_in, 0, sizeof(float) * (size_t)rows_in * n_in_planes, stream));
    return SCN_OK;
  }
  SCN_REQUIRE(in && d_out, SCN_ERR_BAD_ARG, "null features");

  // ---- d_bias -------------------------------------------------------------------------------------
  if (d_bias) {
    const int chunks = n_chunks(rows_out);
    const long long chunk_rows = ceil_div(rows_out, chunks);
    Scratch tmp(stream);
    float *partial = nullptr;
    SCN_TRY(tmp.get(&partial, sizeof(float) * (size_t)chunks * n_out_planes));
    SCN_LAUNCH(k_column_sums, dim3((unsigned)ceil_div(n_out_planes, 32), (unsigned)chunks), 256, 0, stream, d_out, rows_out, n_out_planes, chunk_rows, partial);
    SCN_LAUNCH(k_sum_chunks, (unsigned)ceil_div(n_out_planes, 256), 256, 0, stream, partial, chunks, (long long)n_out_planes, d_bias, false);
    SCN_CUDA_CHECK(cudaGetLastError());
  }

  // ---- d_weight -----------------------------------------------------------------------------------
  {
    const long long n_entries = rb.n_out;  // nbr is [K][rb.n_out]
    const bool fma_only = getenv("SCN_DWEIGHT_FMA") && atoi(getenv("SCN_DWEIGHT_FMA")) != 0;
    const char *tile = getenv("SCN_DWEIGHT_TILE");
    if (groups == 1 && !fma_only && !(tile && atoi(tile) == 0) && dweight_tile_supported(in, d_out, rb, cin, cout)) {
      SCN_TRY(rulebook_row_order(rb, rb.nbr, rb.n_out, rb.order, stream));
      g_last_dweight_kernel = SCN_KERNEL_DWEIGHT_TILE;
      SCN_TRY(dweight_tile(in, rows_in, d_out, rows_out, rb, transposed, cin, cout, d_weight, md->flags_dev, stream));
    } else if (groups == 1 && !fma_only && cin <= 3 && cout <= 32 && !transposed && rows_out > 0) {
      g_last_dweight_kernel = SCN_KERNEL_DWEIGHT_THIN;
      SCN_TRY(dweight_thin(in, rows_in, d_out, rows_out, rb.nbr, K, cin, cout, d_weight, md->flags_dev, stream));
    } else if (groups == 1 && !fma_only) {
      decltype(&launch_dweight<1, 1>) const by_side[3][3] = {{launch_dweight<1, 1>, launch_dweight<1, 2>, launch_dweight<1, 3>},
                                                             {launch_dweight<2, 1>, launch_dweight<2, 2>, launch_dweight<2, 3>},
                                                             {launch_dweight<3, 1>, launch_dweight<3, 2>, launch_dweight<3, 3>}};
      auto launch = by_side[dweight_side(cin, n_entries) - 1][dweight_side(cout, n_entries) - 1];
      if (cin <= 16) launch = cout <= 32 ? launch_dweight<1, 1, 1> : cout <= 64 ? launch_dweight<1, 2, 1> : launch_dweight<1, 3, 1>;
      g_last_dweight_kernel = SCN_KERNEL_DWEIGHT_MMA;
      SCN_TRY(launch(in, n_in_planes, rows_in, d_out, n_out_planes, rows_out, rb.nbr, n_entries, transposed ? 1 : 0, K, cin,
                     cout, d_weight, md->flags_dev, stream));
    } else {
      g_last_dweight_kernel = SCN_KERNEL_DWEIGHT_FMA;
      const int chunks = n_chunks(n_entries);
      const long long chunk_rows = ceil_div(ceil_div(n_entries, chunks), 32) * 32;
      Scratch tmp(stream);
      float *partial = nullptr;
      SCN_TRY(tmp.get(&partial, sizeof(float) * (size_t)chunks * w_elems));
      const int tiles = groups * (int)ceil_div(cin, 32) * (int)ceil_div(cout, 32);
      SCN_LAUNCH(k_conv_dweight, dim3((unsigned)chunks, (unsigned)K, (unsigned)tiles), 256, 0, stream, in, n_in_planes, rows_in, d_out, n_out_planes, rows_out, rb.nbr, n_entries, transposed ? 1 : 0, cin, cout, groups, chunk_rows, partial, md->flags_dev);
      SCN_LAUNCH(k_sum_chunks, (unsigned)ceil_div(w_elems, 256), 256, 0, stream, partial, chunks, w_elems, d_weight, false);
      SCN_CUDA_CHECK(cudaGetLastError());
    }
  }

  // ---- d_input ------------------------------------------------------------------------------------
  if (d_in) {
    Scratch tmp(stream);
    float *wt = nullptr;
    SCN_TRY(tmp.get(&wt, sizeof(float) * (size_t)w_elems));
    // Deconvolution: coarse row <- fine rows, the table as built.  A submanifold rulebook of odd filter sizes is its own
    // transposed one with the offsets in reverse, so that its table and row order serve the backward pass as well.
    const bool mirrored = !transposed && rb.symmetric;
    SCN_LAUNCH(k_transpose_weight, (unsigned)ceil_div(w_elems, 256), 256, 0, stream, weight, wt, (long long)K * groups, cin, cout, mirrored ? groups : 0);
    const bool use_tnbr = !transposed && !mirrored;
    SCN_TRY(conv_forward_table(rb, use_tnbr, d_out, rows_out, d_in, rows_in, wt, nullptr, cout, cin, groups,
                               g_backward_precision.load(), md->flags_dev, stream));
  }
  return SCN_OK;
}

}  // namespace scn

using namespace scn;

extern "C" {

int scn_last_dweight_kernel(void) { return g_last_dweight_kernel; }

int scn_submanifold_convolution_backward(scn_metadata *md, const int64_t *spatial_size, const int64_t *filter_size,
                                         const float *in_features, float *d_in_features,
                                         const float *d_out_features, const float *weight, float *d_weight,
                                         float *d_bias, int n_in_planes, int n_out_planes, int groups,
                                         void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  SCN_REQUIRE(md && spatial_size && filter_size, SCN_ERR_BAD_ARG, "null argument");
  Rulebook *rb = nullptr;
  SCN_TRY(get_submanifold_rulebook(md, spatial_size, filter_size, stream, &rb));
  return run_conv_backward(md, *rb, false, in_features, d_in_features, d_out_features, weight, d_weight, d_bias,
                           n_in_planes, n_out_planes, groups, stream);
}

int scn_convolution_backward(scn_metadata *md, const int64_t *input_size, const int64_t *output_size,
                             const int64_t *filter_size, const int64_t *filter_stride, const float *in_features,
                             float *d_in_features, const float *d_out_features, const float *weight,
                             float *d_weight, float *d_bias, int n_in_planes, int n_out_planes, int groups,
                             void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  SCN_REQUIRE(md && input_size && output_size && filter_size && filter_stride, SCN_ERR_BAD_ARG, "null argument");
  Rulebook *rb = nullptr;
  SCN_TRY(get_strided_rulebook(md, input_size, output_size, filter_size, filter_stride, stream, &rb));
  return run_conv_backward(md, *rb, false, in_features, d_in_features, d_out_features, weight, d_weight, d_bias,
                           n_in_planes, n_out_planes, groups, stream);
}

int scn_rows_affine_backward(const float *in_features, const float *d_out_features, int64_t n_rows, int n_in_planes,
                             int n_out_planes, float *d_weight, float *d_bias, void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  SCN_REQUIRE(n_in_planes >= 1 && n_out_planes >= 1 && d_weight, SCN_ERR_BAD_ARG, "rows_affine_backward: bad arguments");
  SCN_REQUIRE(n_rows >= 0 && n_rows < (1ll << 31), SCN_ERR_UNSUPPORTED, "row count %lld unsupported", (long long)n_rows);
  const long long w_elems = (long long)n_in_planes * n_out_planes;
  if (n_rows == 0) {
    SCN_CUDA_CHECK(cudaMemsetAsync(d_weight, 0, sizeof(float) * (size_t)w_elems, stream));
    if (d_bias) SCN_CUDA_CHECK(cudaMemsetAsync(d_bias, 0, sizeof(float) * (size_t)n_out_planes, stream));
    return SCN_OK;
  }
  SCN_REQUIRE(in_features && d_out_features, SCN_ERR_BAD_ARG, "null features");
  // four waves of CTAs, each at least 16 slabs of 32 rows
  const int tiles = (int)(ceil_div(n_in_planes, 32) * ceil_div(n_out_planes, 32));
  const long long chunks = std::max<long long>(1, std::min<long long>(148 * 32 / tiles, n_rows / 512));
  const long long chunk_rows = ceil_div(ceil_div(n_rows, chunks), 32) * 32;
  const int grid_x = (int)ceil_div(n_rows, chunk_rows);
  Scratch tmp(stream);
  float *partial = nullptr;
  SCN_TRY(tmp.get(&partial, sizeof(float) * (size_t)grid_x * (size_t)(w_elems + n_out_planes)));
  float *bias_partial = partial + (size_t)grid_x * w_elems;
  SCN_LAUNCH(k_conv_dweight, dim3((unsigned)grid_x, 1, (unsigned)tiles), 256, 0, stream, in_features, n_in_planes, (long long)n_rows, d_out_features, n_out_planes, (long long)n_rows, nullptr, (long long)n_rows, 0, n_in_planes, n_out_planes, 1, chunk_rows, partial, nullptr);
  SCN_LAUNCH(k_sum_chunks, (unsigned)ceil_div(w_elems, 32), 32, 0, stream, partial, grid_x, w_elems, d_weight, false);
  if (d_bias) {
    SCN_LAUNCH(k_column_sums, dim3((unsigned)ceil_div(n_out_planes, 32), (unsigned)grid_x), 256, 0, stream, d_out_features, (long long)n_rows, n_out_planes, chunk_rows, bias_partial);
    SCN_LAUNCH(k_sum_chunks, (unsigned)ceil_div(n_out_planes, 32), 32, 0, stream, bias_partial, grid_x, (long long)n_out_planes, d_bias, false);
  }
  SCN_CUDA_CHECK(cudaGetLastError());
  return SCN_OK;
}

int scn_deconvolution_backward(scn_metadata *md, const int64_t *input_size, const int64_t *output_size,
                               const int64_t *filter_size, const int64_t *filter_stride, const float *in_features,
                               float *d_in_features, const float *d_out_features, const float *weight,
                               float *d_weight, float *d_bias, int n_in_planes, int n_out_planes, int groups,
                               void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  SCN_REQUIRE(md && input_size && output_size && filter_size && filter_stride, SCN_ERR_BAD_ARG, "null argument");
  Rulebook *rb = nullptr;
  SCN_TRY(get_strided_rulebook(md, output_size, input_size, filter_size, filter_stride, stream, &rb));
  return run_conv_backward(md, *rb, true, in_features, d_in_features, d_out_features, weight, d_weight, d_bias,
                           n_in_planes, n_out_planes, groups, stream);
}
}
