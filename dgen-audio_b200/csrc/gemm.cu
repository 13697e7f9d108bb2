// Controller layers and optimiser: dense fp32 matmul (+ bias, tanh), its backward, and Adam.
//
// The reference expresses a layer as mul + sumAxis over a broadcast [M,N,K] product on the C backend
// and as 8x8 simdgroup tiles on Metal (Sources/DGen/Tensor.swift:1195-1230, Sources/DGen/Emit+GEMM.swift);
// parameters live on the host and Adam is a per-element Swift loop (Sources/DGenLazy/Optimizers.swift:164-243).
// Here activations, weights, gradients and optimiser state stay in HBM.  The matmul runs on the
// tcgen05 tensor cores in 3xTF32 (tc_gemm.cuh: fp32-grade accuracy, which the gradient tolerance of the
// path -- 1e-3 relative against an fp64 evaluation -- needs; single-pass TF32 would not do), and a
// register-tiled SIMT kernel covers small shapes.
#include <stdlib.h>

#include "common.cuh"
#include "tc_gemm.cuh"

namespace {

// C[M][N] (+)= op(A) * op(B) with 128x128 block tiles, 8-deep k-slices, 8x8 register tiles per thread.
// TA: A is stored [K][M] (use A^T);  TB: B is stored [N][K] (use B^T).
constexpr int BM = 128, BN = 128, BK = 8, TM = 8, TN = 8;

// EPI 0: C = acc ; 1: C = acc + bias[n] ; 2: C = tanh(acc + bias[n])
template <bool TA, bool TB, int EPI>
__global__ void __launch_bounds__(256)
sgemm_kernel(const float *__restrict__ A, const float *__restrict__ B, const float *__restrict__ bias, int M, int N,
             int K, int k_per_split, float *__restrict__ C) {
  dgc_after_previous();
  __shared__ float As[BK][BM + 4];
  __shared__ float Bs[BK][BN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tx = tid % 16, ty = tid / 16;  // 16 x 16 threads, each 8 x 8 outputs
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

  // split-K: slice blockIdx.z of the reduction range goes to its own [M][N] slab of C
  const int k_begin = blockIdx.z * k_per_split;
  const int k_end = min(K, k_begin + k_per_split);
  C += (size_t)blockIdx.z * M * N;
  for (int k0 = k_begin; k0 < k_end; k0 += BK) {
    // stage A tile [BM][BK] and B tile [BK][BN]: 1024 elements each, 4 per thread
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      int idx = tid + e * 256;
      if (!TA) {  // A stored [M][K]: consecutive idx walk k fastest
        int m = idx / BK, k = idx % BK;
        int gm = m0 + m, gk = k0 + k;
        As[k][m] = (gm < M && gk < k_end) ? A[(size_t)gm * K + gk] : 0.0f;
      } else {    // A stored [K][M]: consecutive idx walk m fastest
        int k = idx / BM, m = idx % BM;
        int gm = m0 + m, gk = k0 + k;
        As[k][m] = (gm < M && gk < k_end) ? A[(size_t)gk * M + gm] : 0.0f;
      }
      if (!TB) {  // B stored [K][N]
        int k = idx / BN, n = idx % BN;
        int gn = n0 + n, gk = k0 + k;
        Bs[k][n] = (gn < N && gk < k_end) ? B[(size_t)gk * N + gn] : 0.0f;
      } else {    // B stored [N][K]
        int n = idx / BK, k = idx % BK;
        int gn = n0 + n, gk = k0 + k;
        Bs[k][n] = (gn < N && gk < k_end) ? B[(size_t)gn * K + gk] : 0.0f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; i += 4) {
        float4 v = *reinterpret_cast<const float4 *>(&As[k][ty * 4 + i * 16]);  // rows ty*4 + {0..3} + i*16... see below
        a[i] = v.x; a[i + 1] = v.y; a[i + 2] = v.z; a[i + 3] = v.w;
      }
#pragma unroll
      for (int j = 0; j < TN; j += 4) {
        float4 v = *reinterpret_cast<const float4 *>(&Bs[k][tx * 4 + j * 16]);
        b[j] = v.x; b[j + 1] = v.y; b[j + 2] = v.z; b[j + 3] = v.w;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
  // thread (ty, tx) owns rows m0 + ty*4 + {0..3} and m0 + 64 + ty*4 + {0..3}; same pattern for columns
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    int gm = m0 + ty * 4 + (i & 3) + (i >> 2) * 64;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      int gn = n0 + tx * 4 + (j & 3) + (j >> 2) * 64;
      if (gn >= N) continue;
      float v = acc[i][j];
      if (EPI >= 1) v += bias[gn];
      if (EPI == 2) v = tanhf(v);
      C[(size_t)gm * N + gn] = v;
    }
  }
}

// C[m][n] = sum_z part[z][m][n], z ascending: fixed order, bit-reproducible
__global__ void splitk_reduce_kernel(const float *__restrict__ part, size_t mn, int splits, float *__restrict__ C) {
  dgc_after_previous();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= mn) return;
  float acc = 0.0f;
  for (int z = 0; z < splits; ++z) acc += part[(size_t)z * mn + i];
  C[i] = acc;
}

// true unless DGC_GEMM=simt is set in the environment (keeps the SIMT kernel reachable for comparison)
bool use_tensor_cores() {
  static int v = -1;
  if (v < 0) {
    const char *e = getenv("DGC_GEMM");
    v = (e && strcmp(e, "simt") == 0) ? 0 : 1;
  }
  return v == 1;
}

// true when C = A B^T of this shape runs on the persistent short-reduction tensor-core kernel: 32 <= K <= 72, at
// least one full block of 128 columns, A 16-byte aligned (its row tiles are fetched by bulk copies), no more column
// blocks than SMs.  DGC_GEMM_SMALLK=0 keeps such shapes on the general pipeline.
bool smallk_shape(const dgc_ctx *ctx, const float *A, int M, int N, int K) {
  static const bool on = [] {
    const char *e = getenv("DGC_GEMM_SMALLK");
    return !(e && atoi(e) == 0);
  }();
  if (!on || !use_tensor_cores() || (double)M * N * K < (double)(1 << 21) || K < 32 || K > dgtc::SK::KP_MAX ||
      N < dgtc::TBN || (((uintptr_t)A) & 15) != 0)
    return false;
  const int rem = N % dgtc::TBN;
  const int nblk = (rem > 0 && rem <= dgtc::SK::EXTRA_MAX) ? N / dgtc::TBN : dgc_div_up(N, dgtc::TBN);
  return nblk <= ctx->sm_count;
}

// 64 x 64 tiles of the output that the chip takes at once
bool few_tiles(const dgc_ctx *ctx, int M, int N) {
  return (int64_t)dgc_div_up(M, 64) * dgc_div_up(N, 64) <= ctx->sm_count;
}

// copies of both operands' rows, laid 16-byte aligned ld floats apart
struct AlignedRows {
  const float *A = nullptr, *B = nullptr;
  int ld = 0;
};

template <bool TA, bool TB, int EPI>
int32_t launch_sgemm(dgc_ctx *ctx, const float *A, const float *B, const float *bias, int M, int N, int K, float *C,
                     float *Ct = nullptr, bool *ct_written = nullptr, AlignedRows rows = {}) {
  if (ct_written) *ct_written = false;
  const bool tc = use_tensor_cores() && (double)M * N * K >= (double)(1 << 21) && K >= 32;
  // both operands contiguous along k: rows of 16-byte units (A in tensor memory), or any (4-byte copies, where no pass before
  // has left copies of the rows that are aligned)
  const bool along_k = tc && !TA && TB;
  const bool kk16 = along_k && (K & 3) == 0 && ((((uintptr_t)A) | ((uintptr_t)B)) & 15) == 0;
  const bool kk = kk16 || (along_k && EPI == 0);
  // 128 x 256 tiles: 12 % less shared-memory traffic per flop, but one accumulator and so an epilogue that nothing hides: where
  // a CTA runs one long reduction, the split-K weight gradients
  const bool wide = kk16 && N >= 256 && EPI == 0 && K >= 2048 &&
                    dgc_div_up(N, dgtc::TBN) * dgc_div_up(M, dgtc::TBM) < ctx->sm_count;
  // short reductions (the band -> tap map): persistent CTAs that keep their block of B in shared memory
  if (!TA && TB && EPI == 0 && smallk_shape(ctx, A, M, N, K)) {
    const int rem = N % dgtc::TBN;
    const int n_extra = (rem > 0 && rem <= dgtc::SK::EXTRA_MAX) ? rem : 0;
    const int nblk = n_extra ? N / dgtc::TBN : dgc_div_up(N, dgtc::TBN);
    const int per = std::min(dgc_div_up(M, dgtc::TBM), ctx->sm_count / nblk);
    auto kern = dgtc::tc_gemm_smallk_kernel;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, dgtc::SK::SMEM);
    if (e != cudaSuccess) return dgc_fail(ctx, DGC_ERR_CUDA, "tc_gemm smem opt-in: %s", cudaGetErrorString(e));
    ctx->gemm_paths[2]++;
    dgc_launch(kern, nblk * per, dgtc::SK::THREADS_ALL, dgtc::SK::SMEM, ctx->stream, A, B, M, N, K, nblk, n_extra, per, C,
               ctx->status_dev);
    return DGC_OK;
  }
  const int bm = tc ? dgtc::TBM : BM, bn = wide ? 256 : (tc ? dgtc::TBN : BN);
  const int tiles = dgc_div_up(N, bn) * dgc_div_up(M, bm);
  int splits = 1;
  if (EPI == 0 && tiles < ctx->sm_count && K >= 2048) {
    // few output tiles and a long reduction (weight gradients): split the reduction over blocks -- two per SM for the narrow
    // tiles, one (and never a second, nearly empty wave) for the wide ones
    splits = wide ? ctx->sm_count / tiles : (2 * ctx->sm_count + tiles - 1) / tiles;
    if (splits > K / 256) splits = K / 256;
    if (splits < 1) splits = 1;
  }
  int kps = K;
  float *dst = C;
  if (splits > 1) {
    kps = dgc_div_up(dgc_div_up(K, splits), 32) * 32;
    splits = dgc_div_up(K, kps);
    dst = dgc_ctx_scratch(ctx, (uint64_t)splits * M * N + 4);
    if (!dst) return DGC_ERR_OOM;
  }
  dim3 grid(dgc_div_up(N, bn), dgc_div_up(M, bm), splits);
  // a whole reduction whose 64 x 64 tiles the chip takes at once: smaller tiles beat the pipeline (750 x 128 over 128 k: 10 -> 7 us,
  // 750 x 512 over 512 k: 30 -> 17 us)
  const bool few = tc && splits == 1 && few_tiles(ctx, M, N);
  const bool piped = kk && !few && (splits == 1 || kps % 32 == 0);
  ctx->gemm_paths[piped ? (wide ? 3 : 2) : (tc ? 1 : 0)]++;
  if (piped && !kk16 && rows.A) {
    A = rows.A;
    B = rows.B;
  }
  if (piped && (kk16 || rows.A)) {
    const int ld = kk16 ? K : rows.ld;
    auto kern = dgtc::tc_gemm_ts_kernel<EPI, dgtc::TBN>;
    if constexpr (EPI == 0) {
      if (wide) kern = dgtc::tc_gemm_ts_kernel<EPI, 256>;
    }
    const int smem = wide ? dgtc::TS<256>::SMEM : dgtc::TS<dgtc::TBN>::SMEM;
    CUtensorMap map_a, map_b;
    if (!dgtma::make_map_k16(&map_a, A, M, K, ld, dgtc::TBM) || !dgtma::make_map_k16(&map_b, B, N, K, ld, bn))
      return dgc_fail(ctx, DGC_ERR_CUDA, "tc_gemm: no tensor map for %d x %d x %d", M, N, K);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return dgc_fail(ctx, DGC_ERR_CUDA, "tc_gemm smem opt-in: %s", cudaGetErrorString(e));
    const int64_t items = (int64_t)grid.x * grid.y * grid.z;
    dgc_launch(kern, (unsigned)std::min<int64_t>(items, ctx->sm_count), dgtc::TS<dgtc::TBN>::THREADS_ALL, smem, ctx->stream, map_a,
               map_b, bias, M, N, K, kps, (int)items, dst, splits == 1 ? Ct : nullptr, ctx->status_dev);
    if (ct_written) *ct_written = Ct && splits == 1;
  } else if (piped) {
    auto kern = dgtc::tc_gemm_kk4_kernel;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, dgtc::KK::SMEM);
    if (e != cudaSuccess) return dgc_fail(ctx, DGC_ERR_CUDA, "tc_gemm smem opt-in: %s", cudaGetErrorString(e));
    dgc_launch(kern, grid, dgtc::KK_THREADS, dgtc::KK::SMEM, ctx->stream, A, B, M, N, K, kps, dst, ctx->status_dev);
  } else if (tc) {
    // tensor-core kernel: operand A is K-major in memory when it is NOT transposed ([M][K]);
    // operand B is K-major in memory when it IS given transposed ([N][K])
    // the smallest tile whose grid the chip still takes at once
    auto kern = dgtc::tc_gemm_kernel<!TA, TB, EPI, 128, 128>;
    auto fits = [&](int tm, int tn) {
      if ((int64_t)dgc_div_up(M, tm) * dgc_div_up(N, tn) * splits > ctx->sm_count) return false;
      grid.x = dgc_div_up(N, tn);
      grid.y = dgc_div_up(M, tm);
      return true;
    };
    if (fits(32, 32)) kern = dgtc::tc_gemm_kernel<!TA, TB, EPI, 32, 32>;
    else if (fits(64, 64)) kern = dgtc::tc_gemm_kernel<!TA, TB, EPI, 64, 64>;
    else if (fits(128, 64)) kern = dgtc::tc_gemm_kernel<!TA, TB, EPI, 128, 64>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, dgtc::SMEM_BYTES);
    if (e != cudaSuccess) return dgc_fail(ctx, DGC_ERR_CUDA, "tc_gemm smem opt-in: %s", cudaGetErrorString(e));
    dgc_launch(kern, grid, dgtc::THREADS + 32, dgtc::SMEM_BYTES, ctx->stream, A, B, bias, M, N, K, kps, dst,
               splits == 1 ? Ct : nullptr, ctx->status_dev);
    if (ct_written) *ct_written = Ct && splits == 1;
  } else {
    dgc_launch(sgemm_kernel<TA, TB, EPI>, grid, 256, 0, ctx->stream, A, B, bias, M, N, K, kps, dst);
  }
  if (splits > 1) {
    ctx->launches++;
    size_t mn = (size_t)M * N;
    dgc_launch(splitk_reduce_kernel, dgc_div_up((int64_t)mn, 256), 256, 0, ctx->stream, dst, mn, splits, C);
  }
  return DGC_OK;
}

// out[c][r] = in[r][c] (small weight matrices only), 32 x 32 tiles through shared memory
__global__ void transpose_kernel(const float *__restrict__ in, int R, int Cc, float *__restrict__ out) {
  dgc_after_previous();
  __shared__ float t[32][33];
  int c = blockIdx.x * 32 + threadIdx.x, r0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += 8)
    if (r0 + i < R && c < Cc) t[i][threadIdx.x] = in[(size_t)(r0 + i) * Cc + c];
  __syncthreads();
  int r = r0 + threadIdx.x, c0 = blockIdx.x * 32;
  for (int i = threadIdx.y; i < 32; i += 8)
    if (c0 + i < Cc && r < R) out[(size_t)(c0 + i) * R + r] = t[threadIdx.x][i];
}

// The transposed copy of a tile t[m][n] of 64 x 64 values, out[n][m] (M a multiple of 4, out 16-byte aligned)
constexpr int TT = 64;
__device__ __forceinline__ void store_tile_t(const float (*t)[TT + 1], int m0, int n0, int M, int N, float *__restrict__ out) {
  const int m = (threadIdx.x & 15) * 4;
  if (m0 + m >= M) return;
#pragma unroll
  for (int i = 0; i < TT; i += 16) {
    const int n = i + (threadIdx.x >> 4);
    if (n0 + n < N)
      *reinterpret_cast<float4 *>(out + (size_t)(n0 + n) * M + m0 + m) = make_float4(t[m][n], t[m + 1][n], t[m + 2][n], t[m + 3][n]);
  }
}

// dZ = dC * act'(C) written twice: dZ[m][n] and the transposed copy dZt[n][m] (64 x 64 tiles through shared
// memory), so that the weight-gradient product can read both of its operands along the reduction index.  Four passes
// over the layer and nothing else: 32000 x 512 in 39 us (6.6 TB/s; 61 us in 32 x 32 tiles of single loads).  M a
// multiple of 4; VEC: N too, and every buffer on 16 bytes.
// Rows that are not (165 outputs of the heads) the copy engine cannot fetch: ALIGN (without VEC) lays them ld floats apart in
// dZ_ld for the input gradient, and the blocks past the last tile of dZ do the same for the K rows of W.
template <bool VEC, bool ALIGN>
__global__ void __launch_bounds__(256)
act_bwd_t_kernel(const float *__restrict__ dC, const float *__restrict__ Cv, int M, int N, int act,
                 float *__restrict__ dZ, float *__restrict__ dZt, int ld, float *__restrict__ dZ_ld,
                 const float *__restrict__ W, int K, float *__restrict__ W_ld) {
  dgc_after_previous();
  __shared__ float t[TT][TT + 1];
  const int n0 = blockIdx.x * TT, m0 = blockIdx.y * TT;
  if (ALIGN && m0 >= M) {
    const int n = n0 + (threadIdx.x & 63), k0 = (blockIdx.y - (M + TT - 1) / TT) * TT;
    for (int k = k0 + (threadIdx.x >> 6); k < min(K, k0 + TT); k += 4)
      if (n < N) W_ld[(size_t)k * ld + n] = W[(size_t)k * N + n];
    return;
  }
  if (VEC) {
    const int n = (threadIdx.x & 15) * 4, mr = threadIdx.x >> 4;
    float4 g[4], c[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int m = m0 + 16 * i + mr;
      g[i] = c[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (m < M && n0 + n < N) {
        g[i] = *reinterpret_cast<const float4 *>(dC + (size_t)m * N + n0 + n);
        if (act == 1) c[i] = *reinterpret_cast<const float4 *>(Cv + (size_t)m * N + n0 + n);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int m = 16 * i + mr;
      if (act == 1) {
        g[i].x *= (1.0f - c[i].x * c[i].x);
        g[i].y *= (1.0f - c[i].y * c[i].y);
        g[i].z *= (1.0f - c[i].z * c[i].z);
        g[i].w *= (1.0f - c[i].w * c[i].w);
      }
      if (m0 + m < M && n0 + n < N) *reinterpret_cast<float4 *>(dZ + (size_t)(m0 + m) * N + n0 + n) = g[i];
      t[m][n] = g[i].x;
      t[m][n + 1] = g[i].y;
      t[m][n + 2] = g[i].z;
      t[m][n + 3] = g[i].w;
    }
  } else {
    const int n = threadIdx.x & 63;
    for (int m = threadIdx.x >> 6; m < TT; m += 4) {
      float g = 0.0f;
      if (m0 + m < M && n0 + n < N) {
        const size_t idx = (size_t)(m0 + m) * N + n0 + n;
        g = dC[idx];
        if (act == 1) {
          const float c = Cv[idx];
          g *= (1.0f - c * c);
        }
        dZ[idx] = g;
        if (ALIGN) dZ_ld[(size_t)(m0 + m) * ld + n0 + n] = g;
      }
      t[m][n] = g;
    }
  }
  __syncthreads();
  store_tile_t(t, m0, n0, M, N, dZt);
}

// dZ = dC * (1 - C^2) in place-compatible form (tanh'), or copy when act == 0
__global__ void act_bwd_kernel(const float *__restrict__ dC, const float *__restrict__ Cv, size_t n, int act,
                               float *__restrict__ dZ) {
  dgc_after_previous();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float g = dC[i];
  if (act == 1) {
    float c = Cv[i];
    g *= (1.0f - c * c);
  }
  dZ[i] = g;
}

// the same, four elements per thread (n a multiple of 4, 16-byte aligned buffers)
__global__ void act_bwd4_kernel(const float4 *__restrict__ dC, const float4 *__restrict__ Cv, size_t n4, int act,
                                float4 *__restrict__ dZ) {
  dgc_after_previous();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n4) return;
  float4 g = dC[i];
  if (act == 1) {
    const float4 c = Cv[i];
    g.x *= (1.0f - c.x * c.x);
    g.y *= (1.0f - c.y * c.y);
    g.z *= (1.0f - c.z * c.z);
    g.w *= (1.0f - c.w * c.w);
  }
  dZ[i] = g;
}

// A layer with a handful of inputs (the controller's first layer: K = 2 features) is not a matmul but a streaming
// map: C[m][n] = act(sum_k A[m][k] W[k][n] + bias[n]).  One thread per four consecutive outputs of a row: the K
// inputs of the row are broadcast loads, W and the bias stay in L1, the store is 16 bytes.  Same operation order as
// the tile kernel (k ascending from zero, then the bias, then the library tanh).
template <int KK, int EPI>
__device__ __forceinline__ float4 smallk_quad(const float *__restrict__ A, const float *__restrict__ W,
                                              const float *__restrict__ bias, int N, int m, int n) {
  float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int k = 0; k < KK; ++k) {
    const float a = __ldg(A + (size_t)m * KK + k);
    const float4 w = __ldg(reinterpret_cast<const float4 *>(W + (size_t)k * N + n));
    v[0] = fmaf(a, w.x, v[0]);
    v[1] = fmaf(a, w.y, v[1]);
    v[2] = fmaf(a, w.z, v[2]);
    v[3] = fmaf(a, w.w, v[3]);
  }
  if (EPI >= 1) {
    const float4 bq = __ldg(reinterpret_cast<const float4 *>(bias + n));
    v[0] += bq.x; v[1] += bq.y; v[2] += bq.z; v[3] += bq.w;
  }
  if (EPI == 2) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = tanhf(v[j]);
  }
  return make_float4(v[0], v[1], v[2], v[3]);
}

template <int KK, int EPI>
__global__ void __launch_bounds__(256)
smallk_fwd_kernel(const float *__restrict__ A, const float *__restrict__ W, const float *__restrict__ bias, int M, int N,
                  float *__restrict__ C) {
  dgc_after_previous();
  const int nq = N >> 2;
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)M * nq) return;
  const int m = (int)(idx / nq), n = (int)(idx - (size_t)m * nq) * 4;
  *reinterpret_cast<float4 *>(C + (size_t)m * N + n) = smallk_quad<KK, EPI>(A, W, bias, N, m, n);
}

// With the transposed copy Ct[n][m] that the weight gradient of the next layer reads, in tiles of 64 x 64: 25 us for
// 32000 x 512, 58 us with a transposing pass over C behind it
template <int KK, int EPI>
__global__ void __launch_bounds__(256)
smallk_fwd_t_kernel(const float *__restrict__ A, const float *__restrict__ W, const float *__restrict__ bias, int M, int N,
                    float *__restrict__ C, float *__restrict__ Ct) {
  dgc_after_previous();
  __shared__ float t[TT][TT + 1];
  const int n0 = blockIdx.x * TT, m0 = blockIdx.y * TT, n = (threadIdx.x & 15) * 4;
  if (n0 + n < N) {
#pragma unroll
    for (int i = 0; i < TT; i += 16) {
      const int m = i + (threadIdx.x >> 4);
      if (m0 + m >= M) break;
      const float4 v = smallk_quad<KK, EPI>(A, W, bias, N, m0 + m, n0 + n);
      *reinterpret_cast<float4 *>(C + (size_t)(m0 + m) * N + n0 + n) = v;
      t[m][n] = v.x;
      t[m][n + 1] = v.y;
      t[m][n + 2] = v.z;
      t[m][n + 3] = v.w;
    }
  }
  __syncthreads();
  store_tile_t(t, m0, n0, M, N, Ct);
}

// add(m, value) for the rows m, m + 8, .. below m_end of one column, in order.  Sixteen of them are in flight together, the
// last ones too: one after another those were most of the time of a few hundred rows (750 x 128: 7 -> 5 us).
template <class Add>
__device__ __forceinline__ void sum_rows(const float *__restrict__ column, int N, int m, int m_end, Add add) {
  constexpr int LOADS = 16;
  float d[LOADS];
  for (; m + 8 * (LOADS - 1) < m_end; m += 8 * LOADS) {
#pragma unroll
    for (int j = 0; j < LOADS; ++j) d[j] = column[(size_t)(m + 8 * j) * N];
#pragma unroll
    for (int j = 0; j < LOADS; ++j) add(m + 8 * j, d[j]);
  }
#pragma unroll
  for (int j = 0; j < LOADS; ++j) d[j] = m + 8 * j < m_end ? column[(size_t)(m + 8 * j) * N] : 0.0f;
#pragma unroll
  for (int j = 0; j < LOADS; ++j)
    if (m + 8 * j < m_end) add(m + 8 * j, d[j]);
}

// Its backward: db[n] = sum_m dZ[m][n] and dW[k][n] = sum_m A[m][k] dZ[m][n] from ONE pass over dZ (a matmul
// with a 32000-long reduction and a 2 x 512 output reads dZ at a fraction of the memory rate).  Same two fixed-order
// stages as the bias gradient: block (32 columns x 1024 rows) -> part[chunk][1 + KK][n], then the chunks in order.
template <int KK>
__global__ void __launch_bounds__(256)
smallk_grad_kernel(const float *__restrict__ A, const float *__restrict__ dZ, int M, int N, float *__restrict__ part,
                   float *__restrict__ db, float *__restrict__ dW) {
  dgc_after_previous();
  __shared__ float sh[KK + 1][8][33];
  __shared__ float as[1024 * KK];          // the chunk's rows of A: one coalesced read, then broadcast loads
  const int lane = threadIdx.x & 31, col = blockIdx.x * 32 + lane, rg = threadIdx.x >> 5;
  const int m_begin = blockIdx.y * 1024, m_end = min(M, m_begin + 1024);
  for (int i = threadIdx.x; i < (m_end - m_begin) * KK; i += 256) as[i] = A[(size_t)m_begin * KK + i];
  __syncthreads();
  float acc[KK + 1];
#pragma unroll
  for (int q = 0; q <= KK; ++q) acc[q] = 0.0f;
  if (col < N) {
    sum_rows(dZ + col, N, m_begin + rg, m_end, [&](int m, float d) {
      acc[0] += d;
#pragma unroll
      for (int k = 0; k < KK; ++k) acc[1 + k] = fmaf(as[(m - m_begin) * KK + k], d, acc[1 + k]);
    });
  }
#pragma unroll
  for (int q = 0; q <= KK; ++q) sh[q][rg][lane] = acc[q];
  __syncthreads();
  if (rg == 0 && col < N) {
#pragma unroll
    for (int q = 0; q <= KK; ++q) {
      float t = 0.0f;
#pragma unroll
      for (int r = 0; r < 8; ++r) t += sh[q][r][lane];
      if (gridDim.y > 1) part[((size_t)blockIdx.y * (KK + 1) + q) * N + col] = t;
      else if (q > 0) dW[(size_t)(q - 1) * N + col] = t;   // one chunk: the sums are complete
      else if (db) db[col] = t;
    }
  }
}

// db (may be null) and dW from the chunk sums, chunks in index order
__global__ void smallk_grad_reduce_kernel(const float *__restrict__ part, int chunks, int KK, int N, float *__restrict__ db,
                                          float *__restrict__ dW) {
  dgc_after_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (KK + 1) * N) return;
  const int q = i / N, col = i - q * N;
  float t = 0.0f;
  for (int c = 0; c < chunks; ++c) t += part[((size_t)c * (KK + 1) + q) * N + col];
  if (q == 0) {
    if (db) db[col] = t;
  } else
    dW[(size_t)(q - 1) * N + col] = t;
}

// db[n] = sum_m dZ[m][n].  Stage 1: block (32 columns x 1024 rows) sums its rows in a fixed order into
// part[chunk][n]; stage 2 adds the chunks in index order: bit-reproducible.
__global__ void __launch_bounds__(256)
bias_grad_kernel(const float *__restrict__ dZ, int M, int N, float *__restrict__ part) {
  dgc_after_previous();
  __shared__ float sh[8][33];
  const int col = blockIdx.x * 32 + (threadIdx.x & 31), rg = threadIdx.x >> 5;
  const int m_begin = blockIdx.y * 1024, m_end = min(M, m_begin + 1024);
  float acc = 0.0f;
  if (col < N)
    sum_rows(dZ + col, N, m_begin + rg, m_end, [&](int, float d) { acc += d; });
  sh[rg][threadIdx.x & 31] = acc;
  __syncthreads();
  if (rg == 0 && col < N) {
    float t = 0.0f;
#pragma unroll
    for (int r = 0; r < 8; ++r) t += sh[r][threadIdx.x & 31];
    part[(size_t)blockIdx.y * N + col] = t;
  }
}

__global__ void bias_grad_reduce_kernel(const float *__restrict__ part, int chunks, int N, float *__restrict__ db) {
  dgc_after_previous();
  int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= N) return;
  float t = 0.0f;
  for (int c = 0; c < chunks; ++c) t += part[(size_t)c * N + col];
  db[col] = t;
}

__global__ void adam_kernel(float *__restrict__ theta, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, size_t n, float lr, float b1, float b2, float eps, float c1,
                            float c2) {
  dgc_after_previous();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  // operation order of Optimizers.swift:188-203
  float gi = g[i];
  float mi = __fadd_rn(__fmul_rn(b1, m[i]), __fmul_rn(1.0f - b1, gi));
  float vi = __fadd_rn(__fmul_rn(b2, v[i]), __fmul_rn(__fmul_rn(1.0f - b2, gi), gi));
  m[i] = mi;
  v[i] = vi;
  float mh = __fdiv_rn(mi, c1), vh = __fdiv_rn(vi, c2);
  theta[i] = __fsub_rn(theta[i], __fdiv_rn(__fmul_rn(lr, mh), __fadd_rn(__fsqrt_rn(vh), eps)));
}

}  // namespace

bool dgc_linear_bwd_reads_t(int64_t M, int64_t K, int64_t N) {
  return use_tensor_cores() && (M & 3) == 0 && (double)M * N * K >= (double)(1 << 24);
}

bool dgc_gemm_nt_persistent(const dgc_ctx *ctx, const float *a, int M, int N, int K) { return smallk_shape(ctx, a, M, N, K); }

// C[M][N] = A[M][K] * B[N][K]^T, no epilogue (used for the band -> tap map)
int32_t dgc_gemm_nt(dgc_ctx *ctx, const float *a, const float *b, int M, int N, int K, float *c) {
  int32_t rc = launch_sgemm<false, true, 0>(ctx, a, b, nullptr, M, N, K, c);
  if (rc != DGC_OK) return rc;
  ctx->launches++;
  return dgc_check_launch(ctx, "gemm_nt");
}

DGC_EXPORT int32_t dgc_linear_fwd(dgc_ctx *ctx, const float *a_dev, const float *w_dev, const float *bias_dev,
                                  int32_t M, int32_t K, int32_t N, int32_t act, float *c_dev, float *ct_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, a_dev && w_dev && c_dev, "null pointer");
  DGC_REQUIRE(ctx, M > 0 && K > 0 && N > 0, "size out of range");
  DGC_REQUIRE(ctx, act == 0 || act == 1, "act must be 0 (none) or 1 (tanh)");
  DGC_REQUIRE(ctx, act == 0 || bias_dev, "tanh layers need a bias");
  int32_t rc;
  bool ct_done = false;
  if (use_tensor_cores() && (double)M * N * K >= (double)(1 << 24) && (size_t)K * N <= (4u << 20) && (K & 3) == 0) {
    // The weight matrix is small next to the activations: transpose it once so that BOTH operands of the
    // tensor-core kernel are contiguous along k (vector loads straight into the K-major layout).
    if (!ctx->wt_buf || ctx->wt_floats < (uint64_t)K * N) {
      if (ctx->wt_buf) {
        cudaStreamSynchronize(ctx->stream);
        cudaFree(ctx->wt_buf);
        ctx->buffer_generation++;
        ctx->wt_buf = nullptr;
      }
      DGC_CUDA(ctx, cudaMalloc(&ctx->wt_buf, (size_t)K * N * sizeof(float)));
      ctx->wt_floats = (uint64_t)K * N;
    }
    dgc_launch(transpose_kernel, dim3(dgc_div_up(N, 32), dgc_div_up(K, 32)), dim3(32, 8), 0, ctx->stream, w_dev, K, N,
               ctx->wt_buf);
    DGC_LAUNCHED(ctx, "transpose_w");
    if (act == 1) rc = launch_sgemm<false, true, 2>(ctx, a_dev, ctx->wt_buf, bias_dev, M, N, K, c_dev, ct_dev, &ct_done);
    else if (bias_dev) rc = launch_sgemm<false, true, 1>(ctx, a_dev, ctx->wt_buf, bias_dev, M, N, K, c_dev, ct_dev, &ct_done);
    else rc = launch_sgemm<false, true, 0>(ctx, a_dev, ctx->wt_buf, nullptr, M, N, K, c_dev, ct_dev, &ct_done);
  } else if (K <= 4 && (N & 3) == 0 && ((((uintptr_t)w_dev) | ((uintptr_t)c_dev) | ((uintptr_t)bias_dev)) & 15) == 0) {
    // a handful of inputs: the streaming map
    const int64_t work = (int64_t)M * (N >> 2);
    ct_done = ct_dev && (M & 3) == 0 && (((uintptr_t)ct_dev) & 15) == 0 && dgc_div_up(M, TT) <= 65535;
#define DGC_SMALLK_EPI(KKV, EPI, BIAS)                                                                                \
  do {                                                                                                               \
    if (ct_done)                                                                                                     \
      dgc_launch(smallk_fwd_t_kernel<KKV, EPI>, dim3(dgc_div_up(N, TT), dgc_div_up(M, TT)), 256, 0, ctx->stream, \
          a_dev, w_dev, BIAS, M, N, c_dev, ct_dev);                                                                  \
    else                                                                                                             \
      dgc_launch(smallk_fwd_kernel<KKV, EPI>, (unsigned)dgc_div_up(work, 256), 256, 0, ctx->stream, a_dev, w_dev, BIAS, M, N, \
                 c_dev);                                                                                              \
  } while (0)
#define DGC_SMALLK_FWD(KKV)                                                                                           \
  do {                                                                                                               \
    if (act == 1) DGC_SMALLK_EPI(KKV, 2, bias_dev);                                                                  \
    else if (bias_dev) DGC_SMALLK_EPI(KKV, 1, bias_dev);                                                             \
    else DGC_SMALLK_EPI(KKV, 0, nullptr);                                                                            \
  } while (0)
    if (K == 1) DGC_SMALLK_FWD(1);
    else if (K == 2) DGC_SMALLK_FWD(2);
    else if (K == 3) DGC_SMALLK_FWD(3);
    else DGC_SMALLK_FWD(4);
#undef DGC_SMALLK_FWD
#undef DGC_SMALLK_EPI
    rc = DGC_OK;
  } else
  if (act == 1) rc = launch_sgemm<false, false, 2>(ctx, a_dev, w_dev, bias_dev, M, N, K, c_dev);
  else if (bias_dev) rc = launch_sgemm<false, false, 1>(ctx, a_dev, w_dev, bias_dev, M, N, K, c_dev);
  else rc = launch_sgemm<false, false, 0>(ctx, a_dev, w_dev, nullptr, M, N, K, c_dev);
  if (rc != DGC_OK) return rc;
  DGC_LAUNCHED(ctx, "linear_fwd");
  if (ct_dev && !ct_done) {  // the matmul kernel that ran has no transposed store: one extra pass
    dgc_launch(transpose_kernel, dim3(dgc_div_up(N, 32), dgc_div_up(M, 32)), dim3(32, 8), 0, ctx->stream, c_dev, M, N, ct_dev);
    DGC_LAUNCHED(ctx, "transpose_c");
  }
  return DGC_OK;
}

static int32_t linear_bwd_bias(dgc_ctx *ctx, const float *dz_dev, int32_t M, int32_t N, float *dbias_dev) {
  const int chunks = dgc_div_up(M, 1024);
  float *part = dgc_ctx_scratch(ctx, (uint64_t)chunks * N + 4);
  if (!part) return DGC_ERR_OOM;
  dgc_launch(bias_grad_kernel, dim3(dgc_div_up(N, 32), chunks), 256, 0, ctx->stream, dz_dev, M, N, chunks > 1 ? part : dbias_dev);
  DGC_LAUNCHED(ctx, "bias_grad");
  if (chunks > 1) {   // one chunk is the sum
    dgc_launch(bias_grad_reduce_kernel, dgc_div_up(N, 128), 128, 0, ctx->stream, part, chunks, N, dbias_dev);
    DGC_LAUNCHED(ctx, "bias_grad_reduce");
  }
  return DGC_OK;
}

// A weight gradient reads what dZ and the input are, and nothing waits for it but the optimizer.  beside (optional): when it is
// few tiles' work it runs on the context's side stream, from where the caller's stream stands once dZ is there, and *beside says
// so: whoever asked joins the two before anything reads or overwrites its buffers.  750 rows, 128 wide: 18 us a layer on 16 of the
// SMs beside the 15 of the rest of the layer's backward; the step of 3 x 16001 frames 289 -> 251 us, the loss beside the
// spectral gradient and no second launch for sums of one chunk included.
static int32_t linear_bwd_weights(dgc_ctx *ctx, const float *a_dev, const float *dz_dev, int32_t M, int32_t K, int32_t N,
                                  bool dw_kmajor, float *dw_dev, float *dbias_dev, const float *at_dev);

int32_t dgc_linear_bwd_beside(dgc_ctx *ctx, const float *a_dev, const float *w_dev, const float *c_dev, const float *dc_dev,
                              int32_t M, int32_t K, int32_t N, int32_t act, float *dz_dev, float *da_dev, float *dw_dev,
                              float *dbias_dev, const float *at_dev, bool *beside) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, a_dev && w_dev && dc_dev && dz_dev && dw_dev, "null pointer");
  DGC_REQUIRE(ctx, M > 0 && K > 0 && N > 0, "size out of range");
  DGC_REQUIRE(ctx, act == 0 || (act == 1 && c_dev), "tanh backward needs the layer output");
  const size_t n = (size_t)M * N;
  // With a transposed copy of the layer input at hand, the weight gradient reads both operands along the
  // reduction index m (the asynchronous K-major pipeline): dZ is then written in both orientations.
  const bool dw_kmajor = at_dev && dgc_linear_bwd_reads_t(M, K, N) && (((uintptr_t)at_dev) & 15) == 0;
  AlignedRows rows;
  if (dw_kmajor) {
    // The input gradient dZ W^T reads rows of N floats, too: where they are not on 16 bytes, copies of dZ and W that are (of no
    // use to a few tiles or a short reduction).  N = 165, K = 512, the layer's whole backward with 4-byte copies for this product
    // and with aligned rows: 2000 rows 100 -> 94 us, 8000 rows 85 -> 72, 32000 rows 176 -> 134, 64000 rows 300 -> 224; K = 128:
    // 68.7 -> 60 (8000 rows), 102 -> 93 (32000).  A pass of its own over dZ for the copies: 146 us at 32000 rows, and slower than
    // 4-byte copies at 16000 rows and K = 128 (71 -> 77).
    // The blocks that copy W stand behind dZ's in the grid's second dimension, which ends at 65535.
    bool align = da_dev && (N & 3) && N >= 32 && !few_tiles(ctx, M, K) && !smallk_shape(ctx, dz_dev, M, K, N) &&
                       (int64_t)dgc_div_up(M, TT) + dgc_div_up(K, TT) <= 65535;
    const int ld = (N + 3) & ~3;
    size_t need = n + (size_t)(M + (int64_t)K) * ld;   // M, so n, is a multiple of 4
    align = align && need < ctx->dzt_refused;
    if (!align) need = n;
    if (!ctx->dzt_buf || ctx->dzt_floats < need) {
      if (ctx->dzt_buf) {
        cudaStreamSynchronize(ctx->stream);
        cudaFree(ctx->dzt_buf);
        ctx->buffer_generation++;
        ctx->dzt_buf = nullptr;
      }
      ctx->dzt_floats = 0;
      if (align && cudaMalloc(&ctx->dzt_buf, need * sizeof(float)) != cudaSuccess) {   // no room for the copies: do without
        cudaGetLastError();
        ctx->dzt_refused = need;
        align = false;
        need = n;
      }
      if (!ctx->dzt_buf) DGC_CUDA(ctx, cudaMalloc(&ctx->dzt_buf, need * sizeof(float)));
      ctx->dzt_floats = need;
    }
    float *dz_ld = align ? ctx->dzt_buf + n : nullptr, *w_ld = align ? dz_ld + (size_t)M * ld : nullptr;
    if (align) rows = {dz_ld, w_ld, ld};
    const bool vec = (N & 3) == 0 && ((((uintptr_t)dc_dev) | ((uintptr_t)dz_dev) | (act == 1 ? (uintptr_t)c_dev : 0)) & 15) == 0;
    auto kern = vec ? act_bwd_t_kernel<true, false> : align ? act_bwd_t_kernel<false, true> : act_bwd_t_kernel<false, false>;
    dgc_launch(kern, dim3(dgc_div_up(N, TT), dgc_div_up(M, TT) + (align ? dgc_div_up(K, TT) : 0)), 256, 0, ctx->stream, dc_dev,
               c_dev, M, N, act, dz_dev, ctx->dzt_buf, ld, dz_ld, w_dev, K, w_ld);
  } else {
    const bool vec = (n & 3) == 0 && ((((uintptr_t)dc_dev) | ((uintptr_t)dz_dev) | (act == 1 ? (uintptr_t)c_dev : 0)) & 15) == 0;
    if (vec)
      dgc_launch(act_bwd4_kernel, dgc_div_up((int64_t)(n / 4), 256), 256, 0, ctx->stream,
                 reinterpret_cast<const float4 *>(dc_dev), reinterpret_cast<const float4 *>(c_dev), n / 4, act,
                 reinterpret_cast<float4 *>(dz_dev));
    else
      dgc_launch(act_bwd_kernel, dgc_div_up((int64_t)n, 256), 256, 0, ctx->stream, dc_dev, c_dev, n, act, dz_dev);
  }
  DGC_LAUNCHED(ctx, "act_bwd");
  // the transposed dZ is the context's one copy, which the next layer's call writes: with it everything stays in order
  const bool apart = beside && !dw_kmajor && K > 4 && da_dev && (double)M * N * K < (double)(1 << 24);
  if (beside) *beside = apart;
  int32_t rc = DGC_OK;
  if (apart) {
    const cudaStream_t main_stream = ctx->stream;
    DGC_CUDA(ctx, cudaEventRecord(ctx->fork_ev, main_stream));
    DGC_CUDA(ctx, cudaStreamWaitEvent(ctx->aux_stream, ctx->fork_ev, 0));
    ctx->stream = ctx->aux_stream;
    rc = linear_bwd_weights(ctx, a_dev, dz_dev, M, K, N, dw_kmajor, dw_dev, nullptr, at_dev);
    ctx->stream = main_stream;
  } else {
    rc = linear_bwd_weights(ctx, a_dev, dz_dev, M, K, N, dw_kmajor, dw_dev, dbias_dev, at_dev);
  }
  if (rc != DGC_OK) return rc;
  if (da_dev) {
    // dA[M][K] = dZ[M][N] * W^T[N][K]
    rc = launch_sgemm<false, true, 0>(ctx, dz_dev, w_dev, nullptr, M, K, N, da_dev, nullptr, nullptr, rows);
    if (rc != DGC_OK) return rc;
    DGC_LAUNCHED(ctx, "linear_bwd_da");
  }
  // the side stream has the longer share
  return apart && dbias_dev ? linear_bwd_bias(ctx, dz_dev, M, N, dbias_dev) : DGC_OK;
}

DGC_EXPORT int32_t dgc_linear_bwd(dgc_ctx *ctx, const float *a_dev, const float *w_dev, const float *c_dev,
                                  const float *dc_dev, int32_t M, int32_t K, int32_t N, int32_t act, float *dz_dev,
                                  float *da_dev, float *dw_dev, float *dbias_dev, const float *at_dev) {
  return dgc_linear_bwd_beside(ctx, a_dev, w_dev, c_dev, dc_dev, M, K, N, act, dz_dev, da_dev, dw_dev, dbias_dev, at_dev, nullptr);
}

static int32_t linear_bwd_weights(dgc_ctx *ctx, const float *a_dev, const float *dz_dev, int32_t M, int32_t K, int32_t N,
                                  bool dw_kmajor, float *dw_dev, float *dbias_dev, const float *at_dev) {
  const bool smallk = K <= 4;   // bias and weight gradient from one pass over dZ
  if (smallk) {
    const int chunks = dgc_div_up(M, 1024);
    float *part = dgc_ctx_scratch(ctx, (uint64_t)chunks * (K + 1) * N + 4);
    if (!part) return DGC_ERR_OOM;
    const dim3 grid(dgc_div_up(N, 32), chunks);
    if (K == 1) dgc_launch(smallk_grad_kernel<1>, grid, 256, 0, ctx->stream, a_dev, dz_dev, M, N, part, dbias_dev, dw_dev);
    else if (K == 2) dgc_launch(smallk_grad_kernel<2>, grid, 256, 0, ctx->stream, a_dev, dz_dev, M, N, part, dbias_dev, dw_dev);
    else if (K == 3) dgc_launch(smallk_grad_kernel<3>, grid, 256, 0, ctx->stream, a_dev, dz_dev, M, N, part, dbias_dev, dw_dev);
    else dgc_launch(smallk_grad_kernel<4>, grid, 256, 0, ctx->stream, a_dev, dz_dev, M, N, part, dbias_dev, dw_dev);
    DGC_LAUNCHED(ctx, "smallk_grad");
    if (chunks > 1) {
      dgc_launch(smallk_grad_reduce_kernel, dgc_div_up((K + 1) * N, 128), 128, 0, ctx->stream, part, chunks, K, N, dbias_dev,
                 dw_dev);
      DGC_LAUNCHED(ctx, "smallk_grad_reduce");
    }
  } else if (dbias_dev) {
    const int32_t rc = linear_bwd_bias(ctx, dz_dev, M, N, dbias_dev);
    if (rc != DGC_OK) return rc;
  }
  // dW[K][N] = A^T[K][M] * dZ[M][N]
  int32_t rc = smallk ? DGC_OK : dw_kmajor ? launch_sgemm<false, true, 0>(ctx, at_dev, ctx->dzt_buf, nullptr, K, N, M, dw_dev)
                         : launch_sgemm<true, false, 0>(ctx, a_dev, dz_dev, nullptr, K, N, M, dw_dev);
  if (rc != DGC_OK) return rc;
  if (!smallk) DGC_LAUNCHED(ctx, "linear_bwd_dw");
  return DGC_OK;
}

DGC_EXPORT int32_t dgc_adam_step(dgc_ctx *ctx, float *theta_dev, const float *grad_dev, float *m_dev, float *v_dev,
                                 uint64_t n, int32_t t, float lr, float beta1, float beta2, float eps) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, theta_dev && grad_dev && m_dev && v_dev, "null pointer");
  DGC_REQUIRE(ctx, t >= 1, "t is the 1-based step index");
  if (n == 0) return DGC_OK;
  // bias corrections as the reference computes them: 1 - pow(beta, Float(t)) in single precision
  float c1 = 1.0f - powf(beta1, (float)t), c2 = 1.0f - powf(beta2, (float)t);
  dgc_launch(adam_kernel, dgc_div_up((int64_t)n, 256), 256, 0, ctx->stream, theta_dev, grad_dev, m_dev, v_dev, n, lr, beta1,
             beta2, eps, c1, c2);
  DGC_LAUNCHED(ctx, "adam");
  return DGC_OK;
}

// The same step with the 1-based step index kept in device memory, so that a recorded step (graph.cu) advances it
// on every replay: a one-thread kernel increments *t_dev and evaluates the two bias corrections (in double, then
// rounded: the correctly rounded single-precision power), the update kernel reads them.
namespace {
__global__ void adam_tick_kernel(int32_t *t_dev, float beta1, float beta2, float *corr) {
  dgc_after_previous();
  const int32_t t = *t_dev + 1;
  *t_dev = t;
  corr[0] = 1.0f - (float)pow((double)beta1, (double)t);
  corr[1] = 1.0f - (float)pow((double)beta2, (double)t);
}

__global__ void adam_counted_kernel(float *__restrict__ theta, const float *__restrict__ g, float *__restrict__ m,
                                    float *__restrict__ v, uint64_t n, float lr, float b1, float b2, float eps,
                                    const float *__restrict__ corr) {
  dgc_after_previous();
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float c1 = corr[0], c2 = corr[1];
  float gi = g[i];
  float mi = __fadd_rn(__fmul_rn(b1, m[i]), __fmul_rn(1.0f - b1, gi));
  float vi = __fadd_rn(__fmul_rn(b2, v[i]), __fmul_rn(__fmul_rn(1.0f - b2, gi), gi));
  m[i] = mi;
  v[i] = vi;
  float mh = __fdiv_rn(mi, c1), vh = __fdiv_rn(vi, c2);
  theta[i] = __fsub_rn(theta[i], __fdiv_rn(__fmul_rn(lr, mh), __fadd_rn(__fsqrt_rn(vh), eps)));
}
}  // namespace

DGC_EXPORT int32_t dgc_adam_step_counted(dgc_ctx *ctx, float *theta_dev, const float *grad_dev, float *m_dev,
                                         float *v_dev, uint64_t n, int32_t *t_dev, float *corr_dev, float lr,
                                         float beta1, float beta2, float eps) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, theta_dev && grad_dev && m_dev && v_dev && t_dev && corr_dev, "null pointer");
  dgc_launch(adam_tick_kernel, 1, 1, 0, ctx->stream, t_dev, beta1, beta2, corr_dev);
  DGC_LAUNCHED(ctx, "adam_tick");
  if (n == 0) return DGC_OK;
  dgc_launch(adam_counted_kernel, dgc_div_up((int64_t)n, 256), 256, 0, ctx->stream, theta_dev, grad_dev, m_dev, v_dev, n, lr,
             beta1, beta2, eps, corr_dev);
  DGC_LAUNCHED(ctx, "adam");
  return DGC_OK;
}

DGC_EXPORT int32_t dgc_gemm_path_counts(dgc_ctx *ctx, int64_t *out4) {
  if (!ctx || !out4) return DGC_ERR_INVALID;
  for (int i = 0; i < 4; ++i) out4[i] = ctx->gemm_paths[i];
  return DGC_OK;
}

