// Hop-gated spectral blocks on the sixteen-points-per-thread transforms (windows of 64 points and more): analysis of
// hop pairs, synthesis with the overlap-add kept in registers, and the partitioned convolution along the hops as
// transforms along the hop axis.  16 voices x 480000 samples, 2 s response (N = 2048, hop 1024, 94 partitions), us: analysis 28
// (46 on the eight-point transforms), convolution 66 (245 as a sum over the partitions), synthesis 33 (86 through frames in
// memory); the call 141, from 383.
#pragma once
#include "common.cuh"
#include "fft16.cuh"

namespace dgstft {

using dgfft16::Geo;
using Lay = dgfft16::LayoutFree;
constexpr int THREADS = 128;

enum { SRC_WINDOW = 0, SRC_PARTITION = 1, SRC_ALIGNED = 2 };   // where element i of hop frame h comes from, see stft16_kernel

// The pair of bins (k, N - k) that a thread holds at position (p, t) of a forward transform's registers: the bin k and
// the two values.  t runs to RL - 1, for the thread with local index 0 and p = 0 to RL (its two butterflies pair up
// inside themselves): the same instructions on operands picked by a select, as in the spectral loss.
template <int N, class F>
__device__ __forceinline__ void for_bin_pairs(const float2 (&z)[Geo<N>::PAIRS][2][Geo<N>::RL], int lt, F emit) {
  constexpr int RL = Geo<N>::RL, NBL = Geo<N>::NBL;
  const bool sp = lt == 0;
#pragma unroll
  for (int p = 0; p < Geo<N>::PAIRS; ++p) {
    int ja, jb;
    dgfft16::last_pair<N>(lt, p, ja, jb);
#pragma unroll
    for (int t = 0; t < RL; ++t) {
      float2 zk = z[p][0][t], zn = z[p][1][RL - 1 - t];
      int k = ja + t * NBL;
      if (p == 0) {
        const float2 ks = t <= RL / 2 ? z[0][0][t] : z[0][1][t - RL / 2 - 1];
        const float2 ns = t == 0 ? z[0][0][0] : t < RL / 2 ? z[0][0][RL - t] : t == RL / 2 ? z[0][0][RL / 2]
                                                                                            : z[0][1][RL - 1 - (t - RL / 2 - 1)];
        if (sp) {
          zk = ks;
          zn = ns;
          k = t <= RL / 2 ? t * NBL : NBL / 2 + (t - RL / 2 - 1) * NBL;
        }
      }
      emit(k, zk, zn);
    }
    if (p == 0 && sp) emit(NBL / 2 + (RL / 2 - 1) * NBL, z[0][1][RL / 2 - 1], z[0][1][RL / 2]);
  }
}

// Two hops (2 p, 2 p + 1) of one signal as the real and imaginary part of one transform.
// SRC_WINDOW:    element i of hop frame h = x[h hop - (N-1) + i] window[i]   (bufferView)
// SRC_PARTITION: zero-padded partitions of one impulse response: x[h hop + i], i < hop
// SRC_ALIGNED:   x[h hop + i] window[i], the frames of the overlap-add grid   (adjoint of the scatter)
// out: half spectra [V][H][N/2+1].
// Loads and stores are whole rows of a warp; there is no pass over shared memory but the exchanges of the transform.
template <int N, int SRC>
__global__ void __launch_bounds__(THREADS, 6)
stft16_kernel(const float *__restrict__ x, int T, int hop, int H, const float *__restrict__ window,
              const float2 *__restrict__ tw, float2 *__restrict__ out) {
  dgc_after_previous();
  constexpr int TT = Geo<N>::T, NF = THREADS / TT, PN = Lay::template size<N>(), NB = N / 2 + 1;
  __shared__ float2 sm[NF * PN];
  const int f = threadIdx.x / TT, lt = threadIdx.x % TT, v = blockIdx.y;
  const int h0 = 2 * (blockIdx.x * NF + f), h1 = h0 + 1;
  const float *xv = x + (size_t)v * T;
  const int a0 = SRC == SRC_WINDOW ? h0 * hop - (N - 1) : h0 * hop, a1 = a0 + hop;
  float2 r[16];
  if (SRC != SRC_PARTITION && h1 < H && a0 >= 0 && a1 + N <= T) {
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int i = lt + m * TT;
      const float w = window ? __ldg(window + i) : 1.0f;
      r[m] = make_float2(__ldg(xv + a0 + i) * w, __ldg(xv + a1 + i) * w);
    }
  } else {
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int i = lt + m * TT, t0 = a0 + i, t1 = a1 + i;
      const float w = SRC != SRC_PARTITION && window ? __ldg(window + i) : 1.0f;
      const bool in = SRC != SRC_PARTITION || i < hop;
      r[m] = make_float2(in && h0 < H && t0 >= 0 && t0 < T ? xv[t0] * w : 0.0f, in && h1 < H && t1 >= 0 && t1 < T ? xv[t1] * w : 0.0f);
    }
  }
  float2 z[Geo<N>::PAIRS][2][Geo<N>::RL];
  dgfft16::fft16<N, false, Lay>(r, z, sm + f * PN, sm + f * PN, lt, tw);
  const size_t row0 = (size_t)v * H + h0;
  for_bin_pairs<N>(z, lt, [&](int k, float2 zk, float2 zn) {
    const float2 X0 = make_float2(0.5f * (zk.x + zn.x), 0.5f * (zk.y - zn.y));
    const float2 X1 = make_float2(0.5f * (zk.y + zn.y), 0.5f * (zn.x - zk.x));
    const int kk = k <= N / 2 ? k : N - k;
    float2 *o = out + row0 * NB + kk;
    const float sg = k <= N / 2 ? 1.0f : -1.0f;
    if (h0 < H) o[0] = make_float2(X0.x, sg * X0.y);
    if (h1 < H) o[NB] = make_float2(X1.x, sg * X1.y);
  });
}

// Inverse transform of hop pairs, window, gain, overlap-add.  A thread's elements of a frame are lt + m N/16, and with
// hop = S N/16 a shift by one hop keeps them in the thread: the sixteen running sums of the overlap-add live in registers,
// frames are added oldest first, and after each frame its S oldest sums are final and leave as whole rows.  The threads of
// a transform walk `run` hop pairs of one signal; the pairs before them that still reach into their first hop are
// transformed again.  S = 0: any hop, the frames go to out [V][H][N] and another kernel adds them.
// FULL: Y is split re / im [V][H][N], any complex spectrum (its Hermitian part is taken), else half spectra float2.
// out[v][t], t = position on the overlap-add grid + offset; offset -(N-1) is the adjoint of the bufferView gather.
template <int N, bool FULL, int S>
__global__ void __launch_bounds__(THREADS, 4)
istft16_kernel(const float *__restrict__ Y, const float *__restrict__ Yim, int H, int T, const float *__restrict__ window,
               const float2 *__restrict__ tw, float gain, int offset, int accumulate, int run, float *__restrict__ out) {
  dgc_after_previous();
  constexpr int TT = Geo<N>::T, NF = THREADS / TT, PN = Lay::template size<N>(), NB = N / 2 + 1, RL = Geo<N>::RL, NBL = Geo<N>::NBL;
  constexpr int WARM = S ? (16 / (S ? S : 1)) / 2 : 0;       // pairs whose frames reach past their own two hops
  __shared__ float2 sm[2][NF * PN];
  const int f = threadIdx.x / TT, lt = threadIdx.x % TT, v = blockIdx.y;
  const int first = (blockIdx.x * NF + f) * run;
  const float scale = gain * (1.0f / (float)N);               // the gain, its exponent moved
  float acc[16];
#pragma unroll
  for (int m = 0; m < 16; ++m) acc[m] = 0.0f;
  for (int p = first - WARM; p < first + run; ++p) {
    const int h0 = 2 * p, h1 = h0 + 1;
    const bool live0 = h0 >= 0 && h0 < H, live1 = h0 >= 0 && h1 < H;
    float2 z[Geo<N>::PAIRS][2][RL], r[16];
    const size_t row0 = (size_t)v * H + (live0 ? h0 : 0);
    // bins k of hops h0 and h1 as the real and imaginary part of one transform; bin N - k follows from bin k, except in the
    // thread whose butterflies pair up inside themselves
    auto bins = [&](int k, float2 &y0, float2 &y1) {
      y0 = y1 = make_float2(0.f, 0.f);
      if (FULL) {
        const int kn = (N - k) & (N - 1);
        const float *re = Y + row0 * N, *im = Yim + row0 * N;
        if (live0) y0 = make_float2(0.5f * (re[k] + re[kn]), 0.5f * (im[k] - im[kn]));
        if (live1) y1 = make_float2(0.5f * (re[N + k] + re[N + kn]), 0.5f * (im[N + k] - im[N + kn]));
      } else {
        const float2 *y = reinterpret_cast<const float2 *>(Y) + row0 * NB + (k <= N / 2 ? k : N - k);
        if (live0) y0 = y[0];
        if (live1) y1 = y[NB];
        if (k > N / 2) {
          y0.y = -y0.y;
          y1.y = -y1.y;
        }
      }
    };
#pragma unroll
    for (int q = 0; q < Geo<N>::PAIRS; ++q) {
      int ja, jb;
      dgfft16::last_pair<N>(lt, q, ja, jb);
#pragma unroll
      for (int t = 0; t < RL; ++t) {
        float2 y0, y1;
        bins(ja + t * NBL, y0, y1);
        z[q][0][t] = make_float2(y0.x - y1.y, y0.y + y1.x);
        y0.y = -y0.y;
        y1.y = -y1.y;
        if (q == 0 && lt == 0) bins(jb + (RL - 1 - t) * NBL, y0, y1);
        z[q][1][RL - 1 - t] = make_float2(y0.x - y1.y, y0.y + y1.x);
      }
    }
    if (!Geo<N>::THREE) dgfft16::sync_transform<N>();   // the previous pair's last reads of the one buffer in use
    dgfft16::fft16_T<N, true, Lay>(z, r, sm[0] + f * PN, sm[1] + f * PN, lt, tw);
    if (S == 0) {
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const int i = lt + m * TT;
        const float w = window ? __ldg(window + i) * scale : scale;
        if (live0) out[row0 * N + i] = r[m].x * w;
        if (live1) out[row0 * N + N + i] = r[m].y * w;
      }
    } else {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
#pragma unroll
        for (int m = 0; m < 16; ++m) {
          const float w = window ? __ldg(window + lt + m * TT) * scale : scale;
          acc[m] = fmaf(half ? r[m].y : r[m].x, w, acc[m]);
        }
        if (p >= first) {
          const int t0 = (h0 + half) * (S * TT) + offset + lt;
          float *o = out + (size_t)v * T + t0;
#pragma unroll
          for (int m = 0; m < S; ++m)
            if (t0 + m * TT >= 0 && t0 + m * TT < T) o[m * TT] = accumulate ? o[m * TT] + acc[m] : acc[m];
        }
#pragma unroll
        for (int m = 0; m < 16; ++m) acc[m] = m + S < 16 ? acc[(m + S) & 15] : 0.0f;
      }
    }
  }
}

// ---- the partitioned convolution along the hops -----------------------------------------------------------------------
// Per voice and bin the partitioned convolution is a complex convolution ALONG THE HOPS of the window spectra with the K
// partition spectra, Y[h] = sum_j Hs[j] X[h-j]: 8 K operations per element of Y done directly, while transforms of M hops
// (overlap-save, M - K + 1 results each) take 20 M log2 M / (M - K + 1), 240 for the K = 94, M = 256 of a 2 s response.
// A block takes 16 consecutive bins, a transform's M / 16 threads sit 16 apart: the lanes of a half-warp are the 16 bins of
// one hop, so global rows are whole 128-byte lines and every exchange (one buffer per bin, M + 1 elements apart) is free of
// bank conflicts whatever the transform's index pattern.
// Rounding is relative to the loudest hop of a transform; what the convolution makes exactly zero -- results before the
// first non-zero hop and after the last one's tail -- is written as zero.  A value that is infinite or no number would be
// in every result of its transform: a bin with such a result is summed directly instead, so that it stays where the
// convolution has it (and so that products that overflow a transform do not count as such).
constexpr int HOP_BINS = 16;

// sets flags[bin] for the block's bins that hold a value which is infinite or no number; a barrier for the block
__device__ __forceinline__ bool hop_not_finite(const float2 (&x)[16], int *flags, int bin) {
  float m = 0.0f;      // stays 0 over finite values, turns into NaN at one that is not
#pragma unroll
  for (int i = 0; i < 16; ++i) m = fmaf(x[i].x, 0.0f, fmaf(x[i].y, 0.0f, m));
  if (m != 0.0f) flags[bin] = 1;
  __syncthreads();
  return flags[bin] != 0;
}

struct LayoutFlat {
  template <int N> __device__ static __forceinline__ int l1(int i) { return i; }
  template <int N> __device__ static __forceinline__ int l2(int i) { return i; }
};

template <int M>
__device__ __forceinline__ void hop_forward(float2 (&x)[16], float2 (&z)[Geo<M>::PAIRS][2][Geo<M>::RL], float2 *buf, int lt,
                                            const float2 *__restrict__ tw) {
  dgfft16::stage_first<M, false, LayoutFlat>(x, buf, lt);
  __syncthreads();
  if (Geo<M>::THREE) {
    dgfft16::stage_middle_inplace<M, false, LayoutFlat, dgfft16::SyncBlock>(buf, lt, tw);
    __syncthreads();
  }
  dgfft16::stage_last<M, false, LayoutFlat>(buf, z, lt, tw);
}

// from the register layout hop_forward leaves, back to element lt + m M/16
template <int M>
__device__ __forceinline__ void hop_inverse(float2 (&z)[Geo<M>::PAIRS][2][Geo<M>::RL], float2 (&x)[16], float2 *buf, int lt,
                                            const float2 *__restrict__ tw) {
  __syncthreads();
  dgfft16::stage_last_T<M, true, LayoutFlat>(z, buf, lt, tw);
  __syncthreads();
  if (Geo<M>::THREE) {
    dgfft16::stage_middle_T_inplace<M, true, LayoutFlat, dgfft16::SyncBlock>(buf, lt, tw);
    __syncthreads();
  }
  dgfft16::stage_first_T<M, true, LayoutFlat>(buf, x, lt);
}

// Spectrum along the hops of the K partition spectra Hs [K][NB], scaled by 1/M, in the order the threads hold it:
// G[(register 0..15) (M/16) + lt][ceil(NB/16) 16].
template <int M>
__global__ void __launch_bounds__(M)
hop_spectrum_kernel(const float2 *__restrict__ Hs, int K, int NB, const float2 *__restrict__ tw, float2 *__restrict__ G) {
  dgc_after_previous();
  extern __shared__ float2 sm[];
  constexpr int RL = Geo<M>::RL, TT = Geo<M>::T;
  const int bin = threadIdx.x % HOP_BINS, lt = threadIdx.x / HOP_BINS, k = blockIdx.x * HOP_BINS + bin;
  float2 x[16], z[Geo<M>::PAIRS][2][RL];
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int j = lt + m * TT;
    x[m] = k < NB && j < K ? Hs[(size_t)j * NB + k] : make_float2(0.f, 0.f);
  }
  hop_forward<M>(x, z, sm + bin * (M + 1), lt, tw);
  const int stride = gridDim.x * HOP_BINS;
#pragma unroll
  for (int p = 0; p < Geo<M>::PAIRS; ++p)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int t = 0; t < RL; ++t) {
        const int r = (p * 2 + e) * RL + t;
        G[(size_t)(r * TT + lt) * stride + k] = make_float2(z[p][e][t].x * (1.0f / M), z[p][e][t].y * (1.0f / M));
      }
}

// Y[v][h] = sum_j Hs[j] X[v][h-j], or with ADJ sum_j conj(Hs[j]) X[v][h+j], j < K; blockIdx = (bins, segment, voice)
template <int M, bool ADJ>
__global__ void __launch_bounds__(M, M <= 256 ? 512 / M : 1)
hop_convolve_kernel(const float2 *__restrict__ X, const float2 *__restrict__ Hs, const float2 *__restrict__ G, int H, int K, int NB,
                    const float2 *__restrict__ tw, float2 *__restrict__ Y) {
  dgc_after_previous();
  extern __shared__ float2 sm[];
  __shared__ int lo[HOP_BINS], hi[HOP_BINS], direct[HOP_BINS];
  constexpr int RL = Geo<M>::RL, TT = Geo<M>::T;
  const int bin = threadIdx.x % HOP_BINS, lt = threadIdx.x / HOP_BINS, k = blockIdx.x * HOP_BINS + bin;
  const int L = M - K + 1, from = blockIdx.y * L - (ADJ ? 0 : K - 1);
  const size_t base = (size_t)blockIdx.z * H * NB + k;
  if (threadIdx.x < HOP_BINS) {
    lo[threadIdx.x] = M;
    hi[threadIdx.x] = -2 * M;
    direct[threadIdx.x] = 0;
  }
  float2 x[16], z[Geo<M>::PAIRS][2][RL];
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int i = lt + m * TT, h = from + i;
    x[m] = k < NB && h >= 0 && h < H ? __ldg(X + base + (size_t)h * NB) : make_float2(0.f, 0.f);
  }
  unsigned some16 = 0;      // which of the sixteen are not zero
#pragma unroll
  for (int m = 0; m < 16; ++m)
    some16 |= ((__float_as_uint(x[m].x) | __float_as_uint(x[m].y)) & 0x7fffffffu) ? 1u << m : 0u;
  int first = some16 ? lt + (__ffs(some16) - 1) * TT : M, last = some16 ? lt + (31 - __clz(some16)) * TT : -2 * M;
  hop_forward<M>(x, z, sm + bin * (M + 1), lt, tw);
  first = min(first, __shfl_xor_sync(0xffffffffu, first, 16));
  last = max(last, __shfl_xor_sync(0xffffffffu, last, 16));
  if ((threadIdx.x & 16) == 0) {
    atomicMin(&lo[bin], first);
    atomicMax(&hi[bin], last);
  }
  const int stride = gridDim.x * HOP_BINS;
#pragma unroll
  for (int p = 0; p < Geo<M>::PAIRS; ++p)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int t = 0; t < RL; ++t) {
        float2 g = __ldg(G + (size_t)(((p * 2 + e) * RL + t) * TT + lt) * stride + k);
        if (ADJ) g.y = -g.y;
        z[p][e][t] = dgfft::cmul(z[p][e][t], g);
      }
  hop_inverse<M>(z, x, sm + bin * (M + 1), lt, tw);
  if (hop_not_finite(x, direct, bin)) {
    for (int m = 0; m < 16; ++m) {
      const int i = lt + m * TT, h = from + i;
      if (k >= NB || h < 0 || h >= H || (ADJ ? i >= L : i < K - 1)) continue;
      float2 y = make_float2(0.f, 0.f);
      for (int j = 0; j < K && (ADJ ? h + j < H : j <= h); ++j) {
        const float2 a = X[base + (size_t)(ADJ ? h + j : h - j) * NB];
        float2 b = Hs[(size_t)j * NB + k];
        if (ADJ) b.y = -b.y;
        y.x += a.x * b.x - a.y * b.y;
        y.y += a.x * b.y + a.y * b.x;
      }
      Y[base + (size_t)h * NB] = y;
    }
    return;
  }
  const int some = ADJ ? lo[bin] - (K - 1) : lo[bin], until = ADJ ? hi[bin] : hi[bin] + K - 1;
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int i = lt + m * TT, h = from + i;
    if (k < NB && h < H && (ADJ ? i < L : i >= K - 1))
      Y[base + (size_t)h * NB] = i >= some && i <= until ? x[m] : make_float2(0.f, 0.f);
  }
}

// Partial sums over (voice, segment) of conj(X^) U^ along the hops: work items blockIdx.y, + gridDim.y, ...
// P[blockIdx.y][(register) (M/16) + lt][bins].  A segment is L = M - K + 1 hops of X and the M hops of U from the same start.
template <int M>
__global__ void __launch_bounds__(M)
hop_correlate_kernel(const float2 *__restrict__ X, const float2 *__restrict__ U, int V, int H, int K, int NB, int segs,
                     const float2 *__restrict__ tw, float2 *__restrict__ P) {
  dgc_after_previous();
  extern __shared__ float2 sm[];
  constexpr int RL = Geo<M>::RL, TT = Geo<M>::T;
  const int bin = threadIdx.x % HOP_BINS, lt = threadIdx.x / HOP_BINS, k = blockIdx.x * HOP_BINS + bin;
  const int L = M - K + 1;
  float2 *buf = sm + bin * (M + 1);
  float2 acc[Geo<M>::PAIRS][2][RL];
#pragma unroll
  for (int p = 0; p < Geo<M>::PAIRS; ++p)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int t = 0; t < RL; ++t) acc[p][e][t] = make_float2(0.f, 0.f);
  for (int w = blockIdx.y; w < V * segs; w += gridDim.y) {
    const int v = w / segs, from = (w - v * segs) * L;
    const size_t base = (size_t)v * H * NB + k;
    float2 x[16], zx[Geo<M>::PAIRS][2][RL], zu[Geo<M>::PAIRS][2][RL];
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int i = lt + m * TT, h = from + i;
      x[m] = k < NB && i < L && h < H ? __ldg(X + base + (size_t)h * NB) : make_float2(0.f, 0.f);
    }
    __syncthreads();
    hop_forward<M>(x, zx, buf, lt, tw);
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int h = from + lt + m * TT;
      x[m] = k < NB && h < H ? __ldg(U + base + (size_t)h * NB) : make_float2(0.f, 0.f);
    }
    __syncthreads();
    hop_forward<M>(x, zu, buf, lt, tw);
#pragma unroll
    for (int p = 0; p < Geo<M>::PAIRS; ++p)
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int t = 0; t < RL; ++t) {
          const float2 a = zx[p][e][t], b = zu[p][e][t];
          acc[p][e][t].x += a.x * b.x + a.y * b.y;
          acc[p][e][t].y += a.x * b.y - a.y * b.x;
        }
  }
  const int stride = gridDim.x * HOP_BINS;
  float2 *o = P + (size_t)blockIdx.y * M * stride + k;
#pragma unroll
  for (int p = 0; p < Geo<M>::PAIRS; ++p)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int t = 0; t < RL; ++t) o[(size_t)(((p * 2 + e) * RL + t) * TT + lt) * stride] = acc[p][e][t];
}

// Sum of the partial products in a fixed order, back to lags: G[k][bin], k < K
template <int M>
__global__ void __launch_bounds__(M)
hop_lags_kernel(const float2 *__restrict__ P, int parts, const float2 *__restrict__ X, const float2 *__restrict__ U, int V, int H, int K,
                int NB, const float2 *__restrict__ tw, float2 *__restrict__ G) {
  dgc_after_previous();
  extern __shared__ float2 sm[];
  __shared__ int direct[HOP_BINS];
  if (threadIdx.x < HOP_BINS) direct[threadIdx.x] = 0;      // (barriers of the transform before it is used)
  constexpr int RL = Geo<M>::RL, TT = Geo<M>::T;
  const int bin = threadIdx.x % HOP_BINS, lt = threadIdx.x / HOP_BINS, k = blockIdx.x * HOP_BINS + bin;
  const int stride = gridDim.x * HOP_BINS;
  float2 x[16], z[Geo<M>::PAIRS][2][RL];
#pragma unroll
  for (int p = 0; p < Geo<M>::PAIRS; ++p)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int t = 0; t < RL; ++t) z[p][e][t] = make_float2(0.f, 0.f);
#pragma unroll 2
  for (int s = 0; s < parts; ++s)
#pragma unroll
    for (int p = 0; p < Geo<M>::PAIRS; ++p)
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int t = 0; t < RL; ++t) {
          const float2 u = P[((size_t)s * M + ((p * 2 + e) * RL + t) * TT + lt) * stride + k];
          z[p][e][t].x += u.x;
          z[p][e][t].y += u.y;
        }
  hop_inverse<M>(z, x, sm + bin * (M + 1), lt, tw);
  if (hop_not_finite(x, direct, bin)) {
    for (int m = 0; m < 16; ++m) {
      const int j = lt + m * TT;
      if (k >= NB || j >= K) continue;
      float2 g = make_float2(0.f, 0.f);
      for (int v = 0; v < V; ++v)
        for (int h = j; h < H; ++h) {
          const float2 a = X[((size_t)v * H + h - j) * NB + k], b = U[((size_t)v * H + h) * NB + k];
          g.x += a.x * b.x + a.y * b.y;
          g.y += a.x * b.y - a.y * b.x;
        }
      G[(size_t)j * NB + k] = g;
    }
    return;
  }
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int j = lt + m * TT;
    if (k < NB && j < K) G[(size_t)j * NB + k] = make_float2(x[m].x * (1.0f / M), x[m].y * (1.0f / M));
  }
}

}  // namespace dgstft
