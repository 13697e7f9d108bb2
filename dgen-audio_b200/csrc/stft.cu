// Hop-gated spectral blocks: buffer -> FFT (magnitude or half spectrum), partitioned spectral
// multiply-accumulate, IFFT, overlap-add.
//
// The reference gates these on a hop counter inside a per-frame loop (bufferView ring write every
// frame, window gather + host FFT call when the counter reads 0, scatter-add into an output ring:
// Sources/DGen/HigherOps.swift:738-813, Sources/DGen/Emit+FFT.swift:6-62,
// Sources/DGen/Emit+PartitionedConvolution.swift:26-113).  All hop frames are known up front, so
// here every window is gathered straight from the contiguous signal and transformed in shared
// memory, batched over hops x voices; two real windows share one complex transform; overlap-add
// is a gather (each output frame sums the <= N/hop windows that cover it, oldest first, which is
// the order the reference's ring accumulates them).
#include "common.cuh"
#include "fft.cuh"
#include "stft16.cuh"

namespace {

using namespace dgfft;
constexpr int ST_THREADS = 256;

// Pair p of transform slot holds real sequences (2p, 2p+1) of one signal v as re / im.
// SRC 0: bufferView windows of x[v]: element i of hop frame h = x[h*hop - (N-1) + i] * window[i]
// SRC 1: zero-padded partitions of one IR: element i of partition h = ir[h*hop + i], i < hop
// SRC 2: overlap-add aligned frames of x[v]: element i of hop frame h = x[h*hop + i] * window[i]
//        (the adjoint of the overlap-add scatter, used by the backward pass)
// OUT 0: magnitudes [V][H][N/2+1]     OUT 1: half spectra float2 [V][H][N/2+1]
// OUT 2: all bins, split: real parts to out, imaginary to out_im, [V][H][N] (bins above N/2: the conjugate mirror)
template <int N, int SRC, int OUT>
__global__ void __launch_bounds__(ST_THREADS)
stft_kernel(const float *__restrict__ x, int T, int hop, int H, const float *__restrict__ window,
            const float2 *__restrict__ tw, float *__restrict__ out, float *__restrict__ out_im) {
  dgc_after_previous();
  constexpr int G = N / 8, NF = ST_THREADS / G, NB = N / 2 + 1, PN = padded(N);
  __shared__ float2 bufa[NF * PN];
  __shared__ float2 bufb[NF * PN];
  const int tid = threadIdx.x, f = tid / G, lt = tid % G;
  const int v = blockIdx.y;
  const int pair = blockIdx.x * NF + f;
  const int h0 = 2 * pair, h1 = h0 + 1;
  const float *xv = x + (size_t)v * T;
  float2 *a = bufa + f * PN, *bb = bufb + f * PN;
  float2 vin[8];   // a thread's loads (stride G) are its inputs of the first radix-8 stage: kept in registers
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    int i = lt + q * G;
    float w = (SRC != 1 && window) ? __ldg(&window[i]) : 1.0f;
    float2 val = make_float2(0.f, 0.f);
    if (SRC == 0) {
      int t0 = h0 * hop - (N - 1) + i, t1 = h1 * hop - (N - 1) + i;
      if (h0 < H && t0 >= 0 && t0 < T) val.x = xv[t0] * w;
      if (h1 < H && t1 >= 0 && t1 < T) val.y = xv[t1] * w;
    } else if (SRC == 1) {
      int t0 = h0 * hop + i, t1 = h1 * hop + i;
      if (h0 < H && i < hop && t0 < T) val.x = xv[t0];
      if (h1 < H && i < hop && t1 < T) val.y = xv[t1];
    } else {
      int t0 = h0 * hop + i, t1 = h1 * hop + i;
      if (h0 < H && t0 < T) val.x = xv[t0] * w;
      if (h1 < H && t1 < T) val.y = xv[t1] * w;
    }
    vin[q] = val;
  }
  float2 *z = fft_block_regs<N, false>(vin, a, bb, lt, tw);
  // bins 0..N/2 of both sequences
  for (int k = lt; k < NB; k += G) {
    float2 zk = z[pad(k)], zn = z[pad((N - k) & (N - 1))];
    float2 X0 = make_float2(0.5f * (zk.x + zn.x), 0.5f * (zk.y - zn.y));
    float2 X1 = make_float2(0.5f * (zk.y + zn.y), 0.5f * (zn.x - zk.x));
    if (OUT == 0) {
      if (h0 < H) out[((size_t)v * H + h0) * NB + k] = sqrtf(X0.x * X0.x + X0.y * X0.y);
      if (h1 < H) out[((size_t)v * H + h1) * NB + k] = sqrtf(X1.x * X1.x + X1.y * X1.y);
    } else if (OUT == 2) {
      const size_t r0 = ((size_t)v * H + h0) * N, r1 = r0 + N;
      const int kn = (N - k) & (N - 1);
      if (h0 < H) {
        out[r0 + kn] = out[r0 + k] = X0.x;
        out_im[r0 + kn] = -X0.y;
        out_im[r0 + k] = X0.y;
      }
      if (h1 < H) {
        out[r1 + kn] = out[r1 + k] = X1.x;
        out_im[r1 + kn] = -X1.y;
        out_im[r1 + k] = X1.y;
      }
    } else {
      float2 *o = reinterpret_cast<float2 *>(out);
      if (h0 < H) o[((size_t)v * H + h0) * NB + k] = X0;
      if (h1 < H) o[((size_t)v * H + h1) * NB + k] = X1;
    }
  }
}

// Y[v][h][k] = sum_{j < K, j <= h} Hs[j][k] * X[v][h-j][k]   (partitioned spectral MAC, j = 0 first)
// Block: 32 bins x 8 hop groups; each thread carries HPT consecutive hops of one bin.
constexpr int MAC_BINS = 32, MAC_HPT = 4, MAC_HT = 8 * MAC_HPT;

__global__ void __launch_bounds__(256)
partconv_mac_kernel(const float2 *__restrict__ X, const float2 *__restrict__ Hs, int H, int K, int NB,
                    float2 *__restrict__ Y) {
  dgc_after_previous();
  extern __shared__ float2 smem[];
  float2 *hs = smem;                          // [K][MAC_BINS]
  float2 *xs = smem + (size_t)K * MAC_BINS;   // [MAC_HT + K - 1][MAC_BINS], row r <-> hop hb - (K-1) + r
  const int kb = blockIdx.x * MAC_BINS, hb = blockIdx.y * MAC_HT, v = blockIdx.z;
  const int bin = threadIdx.x & 31, hg = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < K * MAC_BINS; i += 256) {
    int j = i / MAC_BINS, kk = i % MAC_BINS;
    hs[i] = (kb + kk < NB) ? Hs[(size_t)j * NB + kb + kk] : make_float2(0.f, 0.f);
  }
  const int rows = MAC_HT + K - 1;
  for (int i = threadIdx.x; i < rows * MAC_BINS; i += 256) {
    int r = i / MAC_BINS, kk = i % MAC_BINS;
    int h = hb - (K - 1) + r;
    xs[i] = (h >= 0 && h < H && kb + kk < NB) ? X[((size_t)v * H + h) * NB + kb + kk] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  float2 acc[MAC_HPT];
#pragma unroll
  for (int u = 0; u < MAC_HPT; ++u) acc[u] = make_float2(0.f, 0.f);
  // hop h = hb + hg*HPT + u reads X row (h - j) -> r = (K-1) + hg*HPT + u - j
  const int rbase = (K - 1) + hg * MAC_HPT;
  float2 win[MAC_HPT];
#pragma unroll
  for (int u = 0; u < MAC_HPT - 1; ++u) win[u] = xs[(size_t)(rbase + u) * MAC_BINS + bin];
  // j = 0 uses rows rbase..rbase+HPT-1; as j grows the window slides down by one row
  win[MAC_HPT - 1] = xs[(size_t)(rbase + MAC_HPT - 1) * MAC_BINS + bin];
  for (int j = 0; j < K; ++j) {
    float2 hv = hs[(size_t)j * MAC_BINS + bin];
#pragma unroll
    for (int u = 0; u < MAC_HPT; ++u) {
      // (ar*br - ai*bi, ar*bi + ai*br) accumulated as the host MAC service does
      acc[u].x += win[u].x * hv.x - win[u].y * hv.y;
      acc[u].y += win[u].x * hv.y + win[u].y * hv.x;
    }
#pragma unroll
    for (int u = MAC_HPT - 1; u > 0; --u) win[u] = win[u - 1];
    int r = rbase - j - 1;
    win[0] = r >= 0 ? xs[(size_t)r * MAC_BINS + bin] : make_float2(0.f, 0.f);
  }
  if (kb + bin < NB) {
#pragma unroll
    for (int u = 0; u < MAC_HPT; ++u) {
      int h = hb + hg * MAC_HPT + u;
      if (h < H) Y[((size_t)v * H + h) * NB + kb + bin] = acc[u];
    }
  }
}

// frames[v][h][i] = Re(IFFT(Y[v][h]))[i] / N * window[i] * gain ; two hops per complex transform
template <int N>
__global__ void __launch_bounds__(ST_THREADS)
istft_kernel(const float2 *__restrict__ Y, int H, const float *__restrict__ window, const float2 *__restrict__ tw,
             float gain, float *__restrict__ frames) {
  dgc_after_previous();
  constexpr int G = N / 8, NF = ST_THREADS / G, NB = N / 2 + 1, PN = padded(N);
  __shared__ float2 bufa[NF * PN];
  __shared__ float2 bufb[NF * PN];
  const int tid = threadIdx.x, f = tid / G, lt = tid % G;
  const int v = blockIdx.y, pair = blockIdx.x * NF + f;
  const int h0 = 2 * pair, h1 = h0 + 1;
  float2 *a = bufa + f * PN, *bb = bufb + f * PN;
  // z = Y0 + i*Y1 with Hermitian extension: Y[N-k] = conj(Y[k])
  float2 vin[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    int k = lt + q * G;
    int ks = k <= N / 2 ? k : N - k;
    float2 y0 = make_float2(0.f, 0.f), y1 = y0;
    if (h0 < H) y0 = Y[((size_t)v * H + h0) * NB + ks];
    if (h1 < H) y1 = Y[((size_t)v * H + h1) * NB + ks];
    if (k > N / 2) { y0.y = -y0.y; y1.y = -y1.y; }
    vin[q] = make_float2(y0.x - y1.y, y0.y + y1.x);
  }
  float2 *z = fft_block_regs<N, true>(vin, a, bb, lt, tw);
  const float invn = 1.0f / (float)N;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    int i = lt + q * G;
    float w = window ? __ldg(&window[i]) : 1.0f;
    float2 val = z[pad(i)];
    if (h0 < H) frames[((size_t)v * H + h0) * N + i] = ((val.x * invn) * w) * gain;
    if (h1 < H) frames[((size_t)v * H + h1) * N + i] = ((val.y * invn) * w) * gain;
  }
}

// out[v][t] (+)= sum over hops h with 0 <= t - h*hop - offset < N of frames[v][h][t - h*hop - offset],
// oldest first.  offset 0: the forward overlap-add; offset -(N-1): the adjoint of the bufferView gather.
__global__ void overlap_add_kernel(const float *__restrict__ frames, int T, int N, int hop, int H, int offset,
                                   int accumulate, float *__restrict__ out) {
  dgc_after_previous();
  int t = blockIdx.x * blockDim.x + threadIdx.x, v = blockIdx.y;
  if (t >= T) return;
  int u = t - offset;            // frame h covers u in [h*hop, h*hop + N)
  int hmax = min(H - 1, u / hop);
  int hmin = u - N < 0 ? 0 : (u - N) / hop + 1;
  float acc = 0.0f;
  for (int h = hmin; h <= hmax; ++h) acc += frames[((size_t)v * H + h) * N + (u - h * hop)];
  size_t o = (size_t)v * T + t;
  out[o] = accumulate ? out[o] + acc : acc;
}

// V[v][m][k] = sum_{j < K, m + j < H} conj(Hs[j][k]) * U[v][m+j][k]: adjoint of the partitioned MAC
__global__ void __launch_bounds__(256)
partconv_mac_adj_kernel(const float2 *__restrict__ U, const float2 *__restrict__ Hs, int H, int K, int NB,
                        float2 *__restrict__ V) {
  dgc_after_previous();
  extern __shared__ float2 smem[];
  float2 *hs = smem;                          // [K][MAC_BINS]
  float2 *us = smem + (size_t)K * MAC_BINS;   // [MAC_HT + K - 1][MAC_BINS], row r <-> hop hb + r
  const int kb = blockIdx.x * MAC_BINS, hb = blockIdx.y * MAC_HT, v = blockIdx.z;
  const int bin = threadIdx.x & 31, hg = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < K * MAC_BINS; i += 256) {
    int j = i / MAC_BINS, kk = i % MAC_BINS;
    hs[i] = (kb + kk < NB) ? Hs[(size_t)j * NB + kb + kk] : make_float2(0.f, 0.f);
  }
  const int rows = MAC_HT + K - 1;
  for (int i = threadIdx.x; i < rows * MAC_BINS; i += 256) {
    int r = i / MAC_BINS, kk = i % MAC_BINS;
    int h = hb + r;
    us[i] = (h < H && kb + kk < NB) ? U[((size_t)v * H + h) * NB + kb + kk] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  float2 acc[MAC_HPT];
#pragma unroll
  for (int u = 0; u < MAC_HPT; ++u) acc[u] = make_float2(0.f, 0.f);
  const int rbase = hg * MAC_HPT;  // hop m = hb + rbase + u reads row rbase + u + j
  for (int j = 0; j < K; ++j) {
    float2 hv = hs[(size_t)j * MAC_BINS + bin];
#pragma unroll
    for (int u = 0; u < MAC_HPT; ++u) {
      float2 x = us[(size_t)(rbase + u + j) * MAC_BINS + bin];
      acc[u].x += x.x * hv.x + x.y * hv.y;   // conj(h) * x
      acc[u].y += x.y * hv.x - x.x * hv.y;
    }
  }
  if (kb + bin < NB) {
#pragma unroll
    for (int u = 0; u < MAC_HPT; ++u) {
      int m = hb + rbase + u;
      if (m < H) V[((size_t)v * H + m) * NB + kb + bin] = acc[u];
    }
  }
}

// G[k][bin] = sum_v sum_h conj(X[v][h-k][bin]) * U[v][h][bin]: gradient of the IR partition spectra.
// block = (32 bins, partition k); 8 thread groups split the (voice, hop) sum, combined in fixed order.  Every partition
// reads both spectra whole, from L2, and that is the bound: 32 signals x 63 hops x 1025 bins, 16 partitions, 57 us with
// IR_LOADS terms in flight per thread (9.3 TB/s), 81 us one after another.
constexpr int IR_LOADS = 8;
__global__ void __launch_bounds__(256)
partconv_ir_grad_kernel(const float2 *__restrict__ X, const float2 *__restrict__ U, int V, int H, int NB,
                        float2 *__restrict__ G) {
  dgc_after_previous();
  __shared__ float2 red[8][33];
  const int bin = blockIdx.x * 32 + (threadIdx.x & 31), k = blockIdx.y, grp = threadIdx.x >> 5;
  float2 acc = make_float2(0.f, 0.f);
  if (bin < NB && k < H) {
    const int hops = H - k, terms = V * hops;
    const float2 *xk = X + bin, *uk = U + (size_t)k * NB + bin;
    int v = grp / hops, h = grp - v * hops;        // term i = v * hops + h reads X[v][h] and U[v][h + k]
    for (int i = grp; i < terms; i += 8 * IR_LOADS) {
      float2 x[IR_LOADS], u[IR_LOADS];
#pragma unroll
      for (int j = 0; j < IR_LOADS; ++j) {
        x[j] = u[j] = make_float2(0.f, 0.f);
        if (i + 8 * j < terms) {
          const size_t at = ((size_t)v * H + h) * NB;
          x[j] = xk[at];
          u[j] = uk[at];
        }
        for (h += 8; h >= hops; h -= hops) ++v;
      }
#pragma unroll
      for (int j = 0; j < IR_LOADS; ++j)
        if (i + 8 * j < terms) {
          acc.x += x[j].x * u[j].x + x[j].y * u[j].y;
          acc.y += x[j].x * u[j].y - x[j].y * u[j].x;
        }
    }
  }
  red[grp][threadIdx.x & 31] = acc;
  __syncthreads();
  if (grp == 0 && bin < NB) {
    float2 t = make_float2(0.f, 0.f);
#pragma unroll
    for (int g2 = 0; g2 < 8; ++g2) {
      t.x += red[g2][threadIdx.x & 31].x;
      t.y += red[g2][threadIdx.x & 31].y;
    }
    G[(size_t)k * NB + bin] = t;
  }
}

// g_ir[k*hop + i] = frames[k][i], i < hop (the zero-padded tail of each partition carries no parameter)
__global__ void take_partitions_kernel(const float *__restrict__ frames, int ir_len, int N, int hop,
                                       float *__restrict__ g_ir) {
  dgc_after_previous();
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ir_len) return;
  int k = t / hop, i = t - k * hop;
  g_ir[t] = frames[(size_t)k * N + i];
}

// half spectra float2 [rows][N/2+1] -> all N bins as split re / im [rows][N] (bins above N/2: the conjugate mirror)
__global__ void half_to_full_kernel(const float2 *__restrict__ half, int64_t rows, int N, float *__restrict__ re,
                                    float *__restrict__ im) {
  dgc_after_previous();
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * N) return;
  const int64_t r = idx / N;
  const int k = (int)(idx - r * N), NB = N / 2 + 1;
  const float2 z = half[r * NB + (k <= N / 2 ? k : N - k)];
  re[idx] = z.x;
  im[idx] = k <= N / 2 ? z.y : -z.y;
}

bool overlap(const float *a, uint64_t n, const float *b, uint64_t m) { return a < b + m && b < a + n; }

// split re / im [rows][N] of ANY complex spectrum -> the half spectrum of its Hermitian part, whose inverse
// transform is the real part of the inverse transform of the whole (the reference keeps only that real part)
__global__ void full_to_half_kernel(const float *__restrict__ re, const float *__restrict__ im, int64_t rows, int N,
                                    float2 *__restrict__ half) {
  dgc_after_previous();
  const int NB = N / 2 + 1;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * NB) return;
  const int64_t r = idx / NB;
  const int k = (int)(idx - r * NB), kn = (N - k) & (N - 1);
  const float *rr = re + r * N, *ii = im + r * N;
  half[idx] = make_float2(0.5f * (rr[k] + rr[kn]), 0.5f * (ii[k] - ii[kn]));
}

template <int N, int SRC, int OUT>
int32_t launch_stft(dgc_ctx *ctx, const float *x, int V, int T, int hop, int H, const float *window, float *out, float *out_im) {
  const float2 *tw = dgc_ctx_twiddles(ctx, N);
  if (!tw) return DGC_ERR_OOM;
  constexpr int NF = ST_THREADS / (N / 8);
  int pairs = (H + 1) / 2;
  dgc_launch(stft_kernel<N, SRC, OUT>, dim3(dgc_div_up(pairs, NF), V), ST_THREADS, 0, ctx->stream, x, T, hop, H, window, tw, out,
             out_im);
  ctx->launches++;
  return dgc_check_launch(ctx, "stft");
}

template <int SRC, int OUT>
int32_t dispatch_stft(dgc_ctx *ctx, int N, const float *x, int V, int T, int hop, int H, const float *window,
                      float *out, float *out_im = nullptr) {
  switch (N) {
#define CASE(NN) case NN: return launch_stft<NN, SRC, OUT>(ctx, x, V, T, hop, H, window, out, out_im);
    CASE(16) CASE(32) CASE(64) CASE(128) CASE(256) CASE(512) CASE(1024) CASE(2048)
#undef CASE
  }
  return dgc_fail(ctx, DGC_ERR_UNSUPPORTED, "FFT size %d (powers of two 16..2048)", N);
}

// The analysis of a long convolution (see in_hop_spectra): half spectra on the sixteen-point transforms
template <int SRC>
int32_t stft16_half(dgc_ctx *ctx, int N, const float *x, int V, int T, int hop, int H, const float *window, float *out) {
  const float2 *tw = dgc_ctx_twiddles(ctx, N);
  if (!tw) return DGC_ERR_OOM;
  const int pairs = (H + 1) / 2;
  switch (N) {
#define CASE(NN) case NN: dgc_launch(dgstft::stft16_kernel<NN, SRC>, dim3(dgc_div_up(pairs, dgstft::THREADS / (NN / 16)), V), dgstft::THREADS, 0, ctx->stream, \
    x, T, hop, H, window, tw, reinterpret_cast<float2 *>(out)); break;
    CASE(64) CASE(128) CASE(256) CASE(512) CASE(1024) CASE(2048)
#undef CASE
  }
  ctx->launches++;
  return dgc_check_launch(ctx, "stft16");
}

// Hop pairs per thread group of the kernels that add frames in registers: the shortest run with which the grid is resident
// at once (per_sm blocks of nf transforms), up to 8: longer runs repeat fewer of the transforms that reach into the next
// one, but leave too few blocks to hide their latency.
int ola_run(const dgc_ctx *ctx, int V, int pairs, int per_sm, int nf) {
  const int run = dgc_div_up((int64_t)V * pairs, (int64_t)ctx->sm_count * per_sm * nf);
  return run > 8 ? 8 : run;
}

// Inverse transforms and overlap-add into out[V][T] on the sixteen-point transforms.  Y: half spectra, or with Yim split
// full spectra.  frames: V H N floats, used where the hop is no 1/1, 1/2, 1/4 or 1/8 of the window, or where out lies in Y.
template <int N>
int32_t launch_istft16_ola(dgc_ctx *ctx, const float *Y, const float *Yim, int V, int H, int T, int hop, const float *window,
                           float gain, int offset, int accumulate, float *frames, float *out, bool in_place) {
  const float2 *tw = dgc_ctx_twiddles(ctx, N);
  if (!tw) return DGC_ERR_OOM;
  constexpr int TT = N / 16, NF = dgstft::THREADS / TT;
  const int pairs = (dgc_div_up((int64_t)T - offset, hop) + 1) / 2, run = ola_run(ctx, V, pairs, 4, NF);
  const dim3 grid(dgc_div_up(dgc_div_up(pairs, run), NF), V);
#define RUN(FULL, SS) dgc_launch(dgstft::istft16_kernel<N, FULL, SS>, grid, dgstft::THREADS, 0, ctx->stream, \
      Y, Yim, H, T, window, tw, gain, offset, accumulate, run, out)
#define STEP(SS) if (!in_place && hop == SS * TT) {                                                                              \
    if (Yim) RUN(true, SS); else RUN(false, SS);                                                                    \
    ctx->launches++;                                                                                                \
    return dgc_check_launch(ctx, "istft_overlap_add");                                                              \
  }
  STEP(8) STEP(4) STEP(2) STEP(16)
#undef STEP
#undef RUN
  const dim3 every(dgc_div_up((H + 1) / 2, NF), V);
  if (Yim) dgc_launch(dgstft::istft16_kernel<N, true, 0>, every, dgstft::THREADS, 0, ctx->stream, Y, Yim, H, T, window, tw, gain,
                      0, 0, 1, frames);
  else dgc_launch(dgstft::istft16_kernel<N, false, 0>, every, dgstft::THREADS, 0, ctx->stream, Y, Yim, H, T, window, tw, gain, 0,
                  0, 1, frames);
  ctx->launches++;
  int32_t rc = dgc_check_launch(ctx, "istft");
  if (rc != DGC_OK) return rc;
  dgc_launch(overlap_add_kernel, dim3(dgc_div_up(T, 256), V), 256, 0, ctx->stream, frames, T, N, hop, H, offset, accumulate, out);
  DGC_LAUNCHED(ctx, "overlap_add");
  return DGC_OK;
}

int32_t istft16_ola(dgc_ctx *ctx, int N, const float *Y, const float *Yim, int V, int H, int T, int hop, const float *window,
                    float gain, int offset, int accumulate, float *frames, float *out, bool in_place = false) {
  switch (N) {
#define CASE(NN) case NN: return launch_istft16_ola<NN>(ctx, Y, Yim, V, H, T, hop, window, gain, offset, accumulate, frames, out, in_place);
    CASE(64) CASE(128) CASE(256) CASE(512) CASE(1024) CASE(2048)
#undef CASE
  }
  return dgc_fail(ctx, DGC_ERR_UNSUPPORTED, "FFT size %d (powers of two 64..2048)", N);
}

// The same on the eight-point transforms, half spectra only, through frames in memory
template <int N>
int32_t launch_istft_ola(dgc_ctx *ctx, const float2 *Y, int V, int H, int T, int hop, const float *window, float gain, int offset,
                         int accumulate, float *frames, float *out) {
  const float2 *tw = dgc_ctx_twiddles(ctx, N);
  if (!tw) return DGC_ERR_OOM;
  constexpr int NF = ST_THREADS / (N / 8);
  dgc_launch(istft_kernel<N>, dim3(dgc_div_up((H + 1) / 2, NF), V), ST_THREADS, 0, ctx->stream, Y, H, window, tw, gain, frames);
  ctx->launches++;
  int32_t rc = dgc_check_launch(ctx, "istft");
  if (rc != DGC_OK) return rc;
  dgc_launch(overlap_add_kernel, dim3(dgc_div_up(T, 256), V), 256, 0, ctx->stream, frames, T, N, hop, H, offset, accumulate, out);
  DGC_LAUNCHED(ctx, "overlap_add");
  return DGC_OK;
}

int32_t istft_ola(dgc_ctx *ctx, int N, const float *Y, int V, int H, int T, int hop, const float *window, float gain, int offset,
                  int accumulate, float *frames, float *out) {
  const float2 *y = reinterpret_cast<const float2 *>(Y);
  switch (N) {
#define CASE(NN) case NN: return launch_istft_ola<NN>(ctx, y, V, H, T, hop, window, gain, offset, accumulate, frames, out);
    CASE(16) CASE(32) CASE(64) CASE(128) CASE(256) CASE(512) CASE(1024) CASE(2048)
#undef CASE
  }
  return dgc_fail(ctx, DGC_ERR_UNSUPPORTED, "FFT size %d (powers of two 16..2048)", N);
}

// The inverse transforms of H rows of half spectra as frames [H][N]
int32_t istft_frames(dgc_ctx *ctx, int N, const float *Y, int H, float gain, float *frames) {
  const float2 *tw = dgc_ctx_twiddles(ctx, N), *y = reinterpret_cast<const float2 *>(Y);
  if (!tw) return DGC_ERR_OOM;
  switch (N) {
#define CASE(NN) case NN: dgc_launch(istft_kernel<NN>, dgc_div_up((H + 1) / 2, ST_THREADS / (NN / 8)), ST_THREADS, 0, ctx->stream, \
    y, H, nullptr, tw, gain, frames); break;
    CASE(16) CASE(32) CASE(64) CASE(128) CASE(256) CASE(512) CASE(1024) CASE(2048)
#undef CASE
  }
  ctx->launches++;
  return dgc_check_launch(ctx, "istft");
}

// Transform size along the hops for K partitions, or 0: the direct sum.  Direct costs 8 K operations per result, the
// transforms about 20 M log2 M / L (L = M - K + 1 results each) plus what a transform pays for its loads, exchanges and
// stores.  Measured (us): convolution 16 x 469 hops x 1025 bins, K = 5: 35 direct, 40 transformed; 12: 52 / 42; 16: 61 / 50;
// 94: 245 / 66.  32 x 63 hops, K = 8: 13 / 20; 12: 16 / 20; 16: 19 / 20.  Correlation (the impulse response's gradient),
// which directly reads both spectra once per partition: 16 x 469, K = 3: 453 / 76; 16: 409 / 54; 32 x 63: 74 to 90 / 40.
// Below the line everything stays on the kernels above, to the last bit: a training step's gradient holds 1 / |X| of bins
// near zero, where a last-bit change of the reverb's output is a different gradient.
constexpr int HOP_MIN_PARTITIONS = 17, HOP_MIN_WINDOWS = 4096;
bool in_hop_spectra(int N, int K) { return N >= 64 && K >= HOP_MIN_PARTITIONS; }
struct HopPlan {
  int M, L, segs;
};
HopPlan hop_plan(int H, int K) {
  HopPlan best = {0, 0, 0};
  double cost = 0.0;
  for (int M = 64, lg = 6; M <= 512; M *= 2, ++lg) {
    const int L = M - K + 1;
    if (L < 1) continue;
    const int segs = dgc_div_up(H, L);
    const double c = (double)segs * M * (lg + 4);
    if (!best.M || c < cost) {
      cost = c;
      best = {M, L, segs};
    }
  }
  return best;
}
int hop_bins(int NB) { return dgc_div_up(NB, dgstft::HOP_BINS) * dgstft::HOP_BINS; }

#define HOP_CASES(M_) switch (M_) { CASE(64) CASE(128) CASE(256) CASE(512) }

int32_t hop_smem(dgc_ctx *ctx, const void *kernel, int M, int *bytes) {
  *bytes = dgstft::HOP_BINS * (M + 1) * (int)sizeof(float2);
  if (*bytes > 48 * 1024) DGC_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, *bytes));
  return DGC_OK;
}

// out[v][h] = sum_j Hs[j] in[v][h-j], or its adjoint sum_j conj(Hs[j]) in[v][h+j]; spec: hop_spectrum_floats of work space
template <bool ADJ>
int32_t convolve_hops(dgc_ctx *ctx, const float *in, const float *hs, int V, int H, int K, int N, float *spec, float *out) {
  const int NB = N / 2 + 1;
  const float2 *in2 = reinterpret_cast<const float2 *>(in), *hs2 = reinterpret_cast<const float2 *>(hs);
  float2 *out2 = reinterpret_cast<float2 *>(out), *g = reinterpret_cast<float2 *>(spec);
  if (in_hop_spectra(N, K)) {
    const HopPlan pl = hop_plan(H, K);
    const float2 *tw = dgc_ctx_twiddles(ctx, pl.M);
    if (!tw) return DGC_ERR_OOM;
    const int groups = dgc_div_up(NB, dgstft::HOP_BINS);
    int bytes = 0;
#define CASE(MM) case MM:                                                                                            \
    if (int32_t rc = hop_smem(ctx, (const void *)dgstft::hop_spectrum_kernel<MM>, MM, &bytes)) return rc;            \
    if (int32_t rc = hop_smem(ctx, (const void *)dgstft::hop_convolve_kernel<MM, ADJ>, MM, &bytes)) return rc;       \
    dgc_launch(dgstft::hop_spectrum_kernel<MM>, groups, MM, bytes, ctx->stream, hs2, K, NB, tw, g);                  \
    DGC_LAUNCHED(ctx, "hop_spectrum");                                                                               \
    dgc_launch(dgstft::hop_convolve_kernel<MM, ADJ>, dim3(groups, pl.segs, V), MM, bytes, ctx->stream, in2, hs2, g, H, K, NB,   \
               tw, out2);                                                                                            \
    break;
    HOP_CASES(pl.M)
#undef CASE
    DGC_LAUNCHED(ctx, "hop_convolve");
    return DGC_OK;
  }
  const int smem = (int)(((size_t)K * MAC_BINS + (size_t)(MAC_HT + K - 1) * MAC_BINS) * sizeof(float2));
  const dim3 grid(dgc_div_up(NB, MAC_BINS), dgc_div_up(H, MAC_HT), V);
  if (ADJ) {
    DGC_CUDA(ctx, cudaFuncSetAttribute(partconv_mac_adj_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    dgc_launch(partconv_mac_adj_kernel, grid, 256, smem, ctx->stream, in2, hs2, H, K, NB, out2);
  } else {
    DGC_CUDA(ctx, cudaFuncSetAttribute(partconv_mac_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    dgc_launch(partconv_mac_kernel, grid, 256, smem, ctx->stream, in2, hs2, H, K, NB, out2);
  }
  DGC_LAUNCHED(ctx, "partconv_mac");
  return DGC_OK;
}

// G[k] = sum over voices and hops of conj(X[h-k]) U[h]; parts: hop_partial_floats of work space
constexpr int HOP_PARTIALS = 1024;    // partial spectra x transform size
int32_t correlate_hops(dgc_ctx *ctx, const float *x, const float *u, int V, int H, int K, int N, float *parts, float *out) {
  const int NB = N / 2 + 1;
  const float2 *x2 = reinterpret_cast<const float2 *>(x), *u2 = reinterpret_cast<const float2 *>(u);
  float2 *out2 = reinterpret_cast<float2 *>(out), *p2 = reinterpret_cast<float2 *>(parts);
  if (in_hop_spectra(N, K) || (K > 2 && (int64_t)V * H >= HOP_MIN_WINDOWS)) {
    const HopPlan pl = hop_plan(H, K);
    const float2 *tw = dgc_ctx_twiddles(ctx, pl.M);
    if (!tw) return DGC_ERR_OOM;
    const int groups = dgc_div_up(NB, dgstft::HOP_BINS), items = V * pl.segs;
    const int n = HOP_PARTIALS / pl.M < items ? HOP_PARTIALS / pl.M : items;
    int bytes = 0;
#define CASE(MM) case MM:                                                                                            \
    if (int32_t rc = hop_smem(ctx, (const void *)dgstft::hop_correlate_kernel<MM>, MM, &bytes)) return rc;           \
    if (int32_t rc = hop_smem(ctx, (const void *)dgstft::hop_lags_kernel<MM>, MM, &bytes)) return rc;                \
    dgc_launch(dgstft::hop_correlate_kernel<MM>, dim3(groups, n), MM, bytes, ctx->stream, x2, u2, V, H, K, NB,       \
               pl.segs, tw, p2);                                                                                     \
    DGC_LAUNCHED(ctx, "hop_correlate");                                                                              \
    dgc_launch(dgstft::hop_lags_kernel<MM>, groups, MM, bytes, ctx->stream, p2, n, x2, u2, V, H, K, NB, tw, out2);     \
    break;
    HOP_CASES(pl.M)
#undef CASE
    DGC_LAUNCHED(ctx, "hop_lags");
    return DGC_OK;
  }
  dgc_launch(partconv_ir_grad_kernel, dim3(dgc_div_up(NB, 32), K), 256, 0, ctx->stream, x2, u2, V, H, NB, out2);
  DGC_LAUNCHED(ctx, "partconv_ir_grad");
  return DGC_OK;
}

uint64_t hop_spectrum_floats(int K, int NB) { return 2ull * 512 * hop_bins(NB) + 4; }
uint64_t hop_partial_floats(int NB) { return 2ull * HOP_PARTIALS * hop_bins(NB) + 4; }

}  // namespace

DGC_EXPORT int32_t dgc_stft_mag(dgc_ctx *ctx, const float *x_dev, int32_t V, int32_t T, int32_t N, int32_t hop,
                                const float *window_dev, float *mags_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, x_dev && mags_dev, "null pointer");
  DGC_REQUIRE(ctx, V > 0 && V <= 65535 && T > 0 && hop > 0, "size out of range");
  DGC_REQUIRE(ctx, dgc_is_pow2(N) && N >= 16 && N <= 2048, "N must be a power of two in 16..2048");
  const int H = dgc_div_up(T, hop);
  return dispatch_stft<0, 0>(ctx, N, x_dev, V, T, hop, H, window_dev, mags_dev);
}

DGC_EXPORT uint64_t dgc_stft_scratch_floats(int32_t V, int32_t T, int32_t N, int32_t hop, int32_t inverse) {
  if (V <= 0 || T <= 0 || N <= 0 || hop <= 0) return 0;
  const uint64_t H = (uint64_t)(T + hop - 1) / hop, NB = N / 2 + 1;
  return ((2 * (uint64_t)V * H * NB + 3) & ~3ull) + (inverse ? (uint64_t)V * H * N : 0) + 16;
}

DGC_EXPORT int32_t dgc_stft_fwd(dgc_ctx *ctx, const float *x_dev, int32_t V, int32_t T, int32_t N, int32_t hop,
                                const float *window_dev, float *scratch_dev, float *re_dev, float *im_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, x_dev && re_dev && im_dev, "null pointer");
  DGC_REQUIRE(ctx, V > 0 && V <= 65535 && T > 0 && hop > 0, "size out of range");
  DGC_REQUIRE(ctx, dgc_is_pow2(N) && N >= 16 && N <= 2048, "N must be a power of two in 16..2048");
  const int H = dgc_div_up(T, hop);
  const uint64_t bins = (uint64_t)V * H * N, samples = (uint64_t)V * T;
  if (!overlap(x_dev, samples, re_dev, bins) && !overlap(x_dev, samples, im_dev, bins))
    return dispatch_stft<0, 2>(ctx, N, x_dev, V, T, hop, H, window_dev, re_dev, im_dev);
  // the spectra take the place of the signal: by way of half spectra in the work space
  float *scr = scratch_dev ? scratch_dev : dgc_ctx_scratch(ctx, dgc_stft_scratch_floats(V, T, N, hop, 0));
  if (!scr) return DGC_ERR_OOM;
  DGC_REQUIRE(ctx, (((uintptr_t)scr) & 7) == 0, "scratch must be 8-byte aligned");
  int32_t rc = dispatch_stft<0, 1>(ctx, N, x_dev, V, T, hop, H, window_dev, scr);
  if (rc != DGC_OK) return rc;
  dgc_launch(half_to_full_kernel, dgc_div_up((int64_t)bins, 256), 256, 0, ctx->stream, reinterpret_cast<const float2 *>(scr),
             (int64_t)V * H, N, re_dev, im_dev);
  DGC_LAUNCHED(ctx, "stft_full_bins");
  return DGC_OK;
}

DGC_EXPORT int32_t dgc_istft_ola(dgc_ctx *ctx, const float *re_dev, const float *im_dev, int32_t V, int32_t T, int32_t N,
                                 int32_t hop, const float *window_dev, float gain, float *scratch_dev,
                                 int32_t accumulate, float *out_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, re_dev && im_dev && out_dev, "null pointer");
  DGC_REQUIRE(ctx, V > 0 && V <= 65535 && T > 0, "size out of range");
  DGC_REQUIRE(ctx, dgc_is_pow2(N) && N >= 16 && N <= 2048, "N must be a power of two in 16..2048");
  DGC_REQUIRE(ctx, hop > 0 && hop <= N, "hop must be in 1..N");
  const int H = dgc_div_up(T, hop), NB = N / 2 + 1;
  const uint64_t bins = (uint64_t)V * H * N, samples = (uint64_t)V * T;
  const bool in_place = overlap(out_dev, samples, re_dev, bins) || overlap(out_dev, samples, im_dev, bins);
  const bool in_registers = N >= 64 && !in_place && (hop == N || hop == N / 2 || hop == N / 4 || hop == N / 8);   // no work space
  float *scr = scratch_dev || in_registers ? scratch_dev : dgc_ctx_scratch(ctx, dgc_stft_scratch_floats(V, T, N, hop, 1));
  if (!scr && !in_registers) return DGC_ERR_OOM;
  DGC_REQUIRE(ctx, (((uintptr_t)scr) & 7) == 0, "scratch must be 8-byte aligned");
  float *frames = scr ? scr + (((size_t)2 * V * H * NB + 3) & ~(size_t)3) : nullptr;
  if (N >= 64)
    return istft16_ola(ctx, N, re_dev, im_dev, V, H, T, hop, window_dev, gain, 0, accumulate, frames, out_dev, in_place);
  const int64_t rows = (int64_t)V * H;
  dgc_launch(full_to_half_kernel, dgc_div_up(rows * NB, 256), 256, 0, ctx->stream, re_dev, im_dev, rows, N,
             reinterpret_cast<float2 *>(scr));
  DGC_LAUNCHED(ctx, "istft_hermitian_part");
  return istft_ola(ctx, N, scr, V, H, T, hop, window_dev, gain, 0, accumulate, frames, out_dev);
}

DGC_EXPORT uint64_t dgc_partconv_scratch_floats(int32_t V, int32_t T, int32_t ir_len, int32_t N, int32_t hop) {
  if (V <= 0 || T <= 0 || ir_len <= 0 || N <= 0 || hop <= 0) return 0;
  uint64_t H = (uint64_t)(T + hop - 1) / hop, K = (uint64_t)(ir_len + hop - 1) / hop, NB = N / 2 + 1;
  // IR spectra, X spectra, Y spectra (float2 each), frames, IR spectra along the hops
  return 2 * K * NB + 2 * (uint64_t)V * H * NB * 2 + (uint64_t)V * H * N + hop_spectrum_floats((int)K, (int)NB) + 64;
}

DGC_EXPORT int32_t dgc_partconv(dgc_ctx *ctx, const float *x_dev, int32_t V, int32_t T, const float *ir_dev,
                                int32_t ir_len, int32_t N, int32_t hop, float gain, float *scratch_dev,
                                int32_t accumulate, float *out_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, x_dev && ir_dev && out_dev, "null pointer");
  DGC_REQUIRE(ctx, V > 0 && V <= 65535 && T > 0 && ir_len > 0, "size out of range");
  DGC_REQUIRE(ctx, dgc_is_pow2(N) && N >= 16 && N <= 2048, "N must be a power of two in 16..2048");
  DGC_REQUIRE(ctx, hop > 0 && hop <= N, "hop must be in 1..N");
  const int H = dgc_div_up(T, hop), K = dgc_div_up(ir_len, hop), NB = N / 2 + 1;
  size_t mac_smem = ((size_t)K * MAC_BINS + (size_t)(MAC_HT + K - 1) * MAC_BINS) * sizeof(float2);
  DGC_REQUIRE(ctx, mac_smem <= 200 * 1024, "impulse response has too many partitions (K <= 380)");
  DGC_REQUIRE(ctx, dgc_div_up(H, MAC_HT) <= 65535, "too many hops");
  float *scr = scratch_dev ? scratch_dev : dgc_ctx_scratch(ctx, dgc_partconv_scratch_floats(V, T, ir_len, N, hop));
  if (!scr) return DGC_ERR_OOM;
  DGC_REQUIRE(ctx, (((uintptr_t)scr) & 15) == 0, "scratch must be 16-byte aligned");
  float *hs = scr;
  float *xs = hs + (((size_t)2 * K * NB + 3) & ~(size_t)3);
  float *ys = xs + (((size_t)2 * V * H * NB + 3) & ~(size_t)3);
  float *frames = ys + (((size_t)2 * V * H * NB + 3) & ~(size_t)3);
  const float *win = dgc_ctx_hann_per(ctx, N);
  if (!win) return DGC_ERR_OOM;
  // partitionIR: FFT of each zero-padded partition (Sources/DGenLazy/SpectralTensorOps.swift:219-243)
  const bool far = in_hop_spectra(N, K);
  int32_t rc = far ? stft16_half<1>(ctx, N, ir_dev, 1, ir_len, hop, K, nullptr, hs)
                   : dispatch_stft<1, 1>(ctx, N, ir_dev, 1, ir_len, hop, K, nullptr, hs);
  if (rc != DGC_OK) return rc;
  // X_h = FFT(hann * window_h)
  rc = far ? stft16_half<0>(ctx, N, x_dev, V, T, hop, H, win, xs) : dispatch_stft<0, 1>(ctx, N, x_dev, V, T, hop, H, win, xs);
  if (rc != DGC_OK) return rc;
  float *spec = frames + (((size_t)V * H * N + 3) & ~(size_t)3);
  rc = convolve_hops<false>(ctx, xs, hs, V, H, K, N, spec, ys);
  if (rc != DGC_OK) return rc;
  return far ? istft16_ola(ctx, N, ys, nullptr, V, H, T, hop, win, gain, 0, accumulate, frames, out_dev)
             : istft_ola(ctx, N, ys, V, H, T, hop, win, gain, 0, accumulate, frames, out_dev);
}

DGC_EXPORT uint64_t dgc_partconv_bwd_scratch_floats(int32_t V, int32_t T, int32_t ir_len, int32_t N, int32_t hop) {
  if (V <= 0 || T <= 0 || ir_len <= 0 || N <= 0 || hop <= 0) return 0;
  uint64_t H = (uint64_t)(T + hop - 1) / hop, K = (uint64_t)(ir_len + hop - 1) / hop, NB = N / 2 + 1;
  // IR spectra + IR-gradient spectra, X, U, V spectra, frames (max of V*H and K frames)
  uint64_t fr = (uint64_t)V * H > K ? (uint64_t)V * H : K;
  // and the IR spectra along the hops or the partial sums of their gradient
  return 4 * K * NB + 3 * (2 * (uint64_t)V * H * NB + 4) + fr * N + hop_spectrum_floats((int)K, (int)NB) +
         hop_partial_floats((int)NB) + 64;
}

// Backward of dgc_partconv (a linear map in x and in ir): g_x = A(ir)^T g_out and/or g_ir.  The reference
// has no backward for partitionedSpectralConvolve (Sources/DGen/Gradients.swift:1156-1164); this is the
// exact adjoint of the forward above, checked against an fp64 evaluation.
DGC_EXPORT int32_t dgc_partconv_bwd(dgc_ctx *ctx, const float *x_dev, int32_t V, int32_t T, const float *ir_dev,
                                    int32_t ir_len, int32_t N, int32_t hop, float gain, const float *g_out_dev,
                                    float *scratch_dev, int32_t accumulate_gx, float *g_x_dev, float *g_ir_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, x_dev && ir_dev && g_out_dev && (g_x_dev || g_ir_dev), "null pointer");
  DGC_REQUIRE(ctx, V > 0 && V <= 65535 && T > 0 && ir_len > 0, "size out of range");
  DGC_REQUIRE(ctx, dgc_is_pow2(N) && N >= 16 && N <= 2048, "N must be a power of two in 16..2048");
  DGC_REQUIRE(ctx, hop > 0 && hop <= N, "hop must be in 1..N");
  const int H = dgc_div_up(T, hop), K = dgc_div_up(ir_len, hop), NB = N / 2 + 1;
  size_t mac_smem = ((size_t)K * MAC_BINS + (size_t)(MAC_HT + K - 1) * MAC_BINS) * sizeof(float2);
  DGC_REQUIRE(ctx, mac_smem <= 200 * 1024, "impulse response has too many partitions (K <= 380)");
  float *scr = scratch_dev ? scratch_dev
                           : dgc_ctx_scratch(ctx, dgc_partconv_bwd_scratch_floats(V, T, ir_len, N, hop));
  if (!scr) return DGC_ERR_OOM;
  DGC_REQUIRE(ctx, (((uintptr_t)scr) & 15) == 0, "scratch must be 16-byte aligned");
  const size_t nh = ((size_t)2 * K * NB + 3) & ~(size_t)3, nx = ((size_t)2 * V * H * NB + 3) & ~(size_t)3;
  float *hs = scr, *gs = hs + nh, *xs = gs + nh, *us = xs + nx, *vs = us + nx, *frames = vs + nx;
  const size_t nf = ((size_t)((int64_t)V * H > K ? (int64_t)V * H : K) * N + 3) & ~(size_t)3;
  float *spec = frames + nf, *parts = spec + ((hop_spectrum_floats(K, NB) + 3) & ~3ull);
  const float *win = dgc_ctx_hann_per(ctx, N);
  if (!win) return DGC_ERR_OOM;
  const bool far = in_hop_spectra(N, K);
  int32_t rc = far ? stft16_half<2>(ctx, N, g_out_dev, V, T, hop, H, win, us)
                   : dispatch_stft<2, 1>(ctx, N, g_out_dev, V, T, hop, H, win, us);   // U_h = FFT(w * g[h*hop ..])
  if (rc != DGC_OK) return rc;
  if (g_x_dev) {
    rc = far ? stft16_half<1>(ctx, N, ir_dev, 1, ir_len, hop, K, nullptr, hs)
             : dispatch_stft<1, 1>(ctx, N, ir_dev, 1, ir_len, hop, K, nullptr, hs);
    if (rc != DGC_OK) return rc;
    rc = convolve_hops<true>(ctx, us, hs, V, H, K, N, spec, vs);
    if (rc != DGC_OK) return rc;
    rc = far ? istft16_ola(ctx, N, vs, nullptr, V, H, T, hop, win, gain, -(N - 1), accumulate_gx, frames, g_x_dev)
             : istft_ola(ctx, N, vs, V, H, T, hop, win, gain, -(N - 1), accumulate_gx, frames, g_x_dev);
    if (rc != DGC_OK) return rc;
  }
  if (g_ir_dev) {
    rc = far ? stft16_half<0>(ctx, N, x_dev, V, T, hop, H, win, xs) : dispatch_stft<0, 1>(ctx, N, x_dev, V, T, hop, H, win, xs);
    if (rc != DGC_OK) return rc;
    rc = correlate_hops(ctx, xs, us, V, H, K, N, parts, gs);
    if (rc != DGC_OK) return rc;
    rc = istft_frames(ctx, N, gs, K, gain, frames);
    if (rc != DGC_OK) return rc;
    dgc_launch(take_partitions_kernel, dgc_div_up(ir_len, 256), 256, 0, ctx->stream, frames, ir_len, N, hop, g_ir_dev);
    DGC_LAUNCHED(ctx, "take_partitions");
  }
  return DGC_OK;
}
