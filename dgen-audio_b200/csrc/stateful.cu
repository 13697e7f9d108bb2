// Stateful ops of the reference whose state is a ring of past inputs or a held value, computed FRAME-PARALLEL:
//
//   tensor delay line      Sources/DGen/HigherOps+DelayLine.swift:33-65, emission Sources/DGen/Emit.swift:331-403
//   spectrum delay (fixed and modulated)
//                          Sources/DGen/HigherOps+SpectrumDelay.swift:20-135, emission Sources/DGen/Emit.swift:405-512
//   latch (sample and hold) Sources/DGen/Definitions.swift:104-113, Sources/DGen/Emit+State.swift:225-262
//   compressor             Sources/DGen/HigherOps.swift:566-651
//   phase vocoder          Sources/DGen/HigherOps+PhaseVocoder.swift:15-88, emission Sources/DGen/Emit+PhaseVocoder.swift:6-118
//
// The reference runs each of them in a sequential block, one frame after the other, because they read and write
// a memory cell.  None of the first three is a true recurrence: a delay line's output at frame n is a gather
// from the INPUT at frames n - k and n - k - 1 (the ring only remembers the input), and a latch's output is the
// input at the most recent trigger frame (a prefix maximum over trigger indices).  So every (frame, lane) element
// is one thread; the ring / held-value cells are read for the frames that reach back before the call and
// rewritten at the end of the call so that consecutive calls continue as the reference's persistent cells do.
// The compressor's attack / release smoother IS a recurrence with a data-dependent coefficient; it is solved for
// all samples of a tile at once (Newton's method on a monotone piecewise-linear map).  The phase
// vocoder carries one value per bin from hop to hop (the synthesis phase): its analysis runs parallel over
// (hop, bin), and so is all of its resynthesis but the sum of the phases.
#include <type_traits>

#include "chain.cuh"
#include "common.cuh"

namespace {

// ---- fractional delay gather ----------------------------------------------------------------------------------
// x [T][W]; ring of R past rows (lane-major [W][R] for the delay line, row-major [R][W] for spectra); head = the
// slot the NEXT row is written to.  The row written n frames into the call sits at slot (head + n) mod R, so the
// row k frames before frame n is x[n - k] when n - k >= 0 and ring slot (head + n - k) mod R otherwise.
template <bool ROW_MAJOR>
__device__ __forceinline__ float delayed_sample(const float *__restrict__ x, const float *__restrict__ ring, int w0,
                                                int64_t n, int k, int e, int W, int R) {
  const int64_t m = n - k;
  if (m >= 0) return x[m * W + e];
  if (!ring) return 0.0f;
  int p = (int)(w0 + m);          // m in [-(R-1), -1]
  if (p < 0) p += R;
  return ROW_MAJOR ? ring[(size_t)p * W + e] : ring[(size_t)e * R + p];
}

// delay_mode: -1 fixed integer delay `fixed_k` (no interpolation), 0 one value for the call, 1 per frame [T],
// 2 per frame and lane [T][W], 3 per lane [W]
template <bool ROW_MAJOR>
__global__ void __launch_bounds__(256)
frac_delay_kernel(const float *__restrict__ x, const float *__restrict__ delay, int delay_mode, int fixed_k, int64_t T,
                  int W, int R, float dmax, const float *__restrict__ ring, const float *__restrict__ head,
                  float *__restrict__ y) {
  dgc_after_previous();
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= T * W) return;
  const int64_t n = idx / W;
  const int e = (int)(idx - n * W);
  const int w0 = head ? (int)head[0] : 0;
  if (delay_mode < 0) {
    y[idx] = delayed_sample<ROW_MAJOR>(x, ring, w0, n, fixed_k, e, W, R);
    return;
  }
  const float d = delay_mode == 0 ? delay[0] : delay_mode == 1 ? delay[n] : delay_mode == 2 ? delay[idx] : delay[e];
  const float dc = d > dmax ? dmax : (d < 0.0f ? 0.0f : d);
  const float kf = floorf(dc), frac = dc - kf;
  const int k = (int)kf;
  // the second tap of the longest delay wraps onto the slot written this frame, as the reference's ring does
  int k1 = k + 1;
  if (k1 >= R) k1 -= R;
  const float s0 = delayed_sample<ROW_MAJOR>(x, ring, w0, n, k, e, W, R);
  const float s1 = delayed_sample<ROW_MAJOR>(x, ring, w0, n, k1, e, W, R);
  y[idx] = fmaf(s1, frac, s0 * (1.0f - frac));
}

// The same gather with FOUR lanes per thread (W a multiple of 4, 16-byte aligned rows): the two taps of a frame are
// 128-bit loads and the result one 128-bit streaming store; only frames that reach back into the ring cell, and
// per-lane delay times, fall back to one access per lane.
template <bool ROW_MAJOR>
__device__ __forceinline__ float4 delayed_sample4(const float *__restrict__ x, const float *__restrict__ ring, int w0,
                                                  int64_t n, int k, int e, int W, int R) {
  const int64_t m = n - k;
  if (m >= 0) return __ldg(reinterpret_cast<const float4 *>(x + m * W + e));
  return make_float4(delayed_sample<ROW_MAJOR>(x, ring, w0, n, k, e, W, R),
                     delayed_sample<ROW_MAJOR>(x, ring, w0, n, k, e + 1, W, R),
                     delayed_sample<ROW_MAJOR>(x, ring, w0, n, k, e + 2, W, R),
                     delayed_sample<ROW_MAJOR>(x, ring, w0, n, k, e + 3, W, R));
}

template <bool ROW_MAJOR>
__global__ void __launch_bounds__(256)
frac_delay4_kernel(const float *__restrict__ x, const float *__restrict__ delay, int delay_mode, int fixed_k, int64_t T,
                   int W, int R, float dmax, const float *__restrict__ ring, const float *__restrict__ head,
                   float *__restrict__ y) {
  dgc_after_previous();
  const int W4 = W >> 2;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, total = T * W4;
  if (idx >= total) return;
  const int64_t n = total <= 0xffffffffLL ? (int64_t)((uint32_t)idx / (uint32_t)W4) : idx / W4;
  const int e = (int)(idx - n * W4) * 4;
  const int w0 = head ? (int)head[0] : 0;
  float4 out;
  if (delay_mode < 0) {
    out = delayed_sample4<ROW_MAJOR>(x, ring, w0, n, fixed_k, e, W, R);
  } else if (delay_mode <= 1) {
    const float d = delay_mode == 0 ? delay[0] : delay[n];
    const float dc = d > dmax ? dmax : (d < 0.0f ? 0.0f : d);
    const float kf = floorf(dc), frac = dc - kf, omf = 1.0f - frac;
    const int k = (int)kf;
    int k1 = k + 1;
    if (k1 >= R) k1 -= R;
    const float4 s0 = delayed_sample4<ROW_MAJOR>(x, ring, w0, n, k, e, W, R);
    const float4 s1 = delayed_sample4<ROW_MAJOR>(x, ring, w0, n, k1, e, W, R);
    out = make_float4(fmaf(s1.x, frac, s0.x * omf), fmaf(s1.y, frac, s0.y * omf), fmaf(s1.z, frac, s0.z * omf),
                      fmaf(s1.w, frac, s0.w * omf));
  } else {
    const float4 d4 = __ldg(reinterpret_cast<const float4 *>(delay_mode == 2 ? delay + n * W + e : delay + e));
    const float dv[4] = {d4.x, d4.y, d4.z, d4.w};
    float o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float dc = dv[j] > dmax ? dmax : (dv[j] < 0.0f ? 0.0f : dv[j]);
      const float kf = floorf(dc), frac = dc - kf;
      const int k = (int)kf;
      int k1 = k + 1;
      if (k1 >= R) k1 -= R;
      const float s0 = delayed_sample<ROW_MAJOR>(x, ring, w0, n, k, e + j, W, R);
      const float s1 = delayed_sample<ROW_MAJOR>(x, ring, w0, n, k1, e + j, W, R);
      o[j] = fmaf(s1, frac, s0 * (1.0f - frac));
    }
    out = make_float4(o[0], o[1], o[2], o[3]);
  }
  __stcs(reinterpret_cast<float4 *>(y + n * W + e), out);
}

template <bool ROW_MAJOR>
static void launch_frac_delay(cudaStream_t st, const float *x, const float *delay, int delay_mode, int fixed_k, int64_t T,
                              int W, int R, float dmax, const float *ring, const float *head, float *y) {
  const bool vec = (W & 3) == 0 && ((((uintptr_t)x) | ((uintptr_t)y) | ((uintptr_t)delay)) & 15) == 0;
  if (vec)
    dgc_launch(frac_delay4_kernel<ROW_MAJOR>, dgc_div_up(T * (W >> 2), 256), 256, 0, st, x, delay, delay_mode, fixed_k, T, W, R,
               dmax, ring, head, y);
  else
    dgc_launch(frac_delay_kernel<ROW_MAJOR>, dgc_div_up(T * W, 256), 256, 0, st, x, delay, delay_mode, fixed_k, T, W, R, dmax,
               ring, head, y);
}

// ring slot p holds, after the call, the last row written to it: frames n = off, off + R, ... < T with
// off = (p - head) mod R; untouched when off >= T
template <bool ROW_MAJOR>
__global__ void ring_update_kernel(const float *__restrict__ x, int64_t T, int W, int R, float *__restrict__ ring,
                                   const float *__restrict__ head) {
  dgc_after_previous();
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)W * R) return;
  // lanes fastest over threads for the row-major ring, slots fastest for the lane-major one: coalesced writes
  const int e = ROW_MAJOR ? (int)(idx % W) : (int)(idx / R);
  const int p = ROW_MAJOR ? (int)(idx / W) : (int)(idx % R);
  const int w0 = (int)head[0];
  int off = p - w0;
  if (off < 0) off += R;
  if (off >= T) return;
  const int64_t last = off + ((T - 1 - off) / R) * R;
  ring[idx] = x[last * W + e];
}

__global__ void head_advance_kernel(float *head, int64_t T, int R) {
  dgc_after_previous();
  const int64_t w0 = (int64_t)head[0];
  head[0] = (float)((w0 + T) % R);
}

// ---- latch ------------------------------------------------------------------------------------------------------
constexpr int LATCH_CHUNK = 128;

__device__ __forceinline__ float cond_at(const float *__restrict__ cond, int cond_mode, int64_t n, int e, int W) {
  return cond_mode == 1 ? cond[n] : cond[n * W + e];
}

// last[c][e] = the last frame of chunk c whose trigger is positive, or -1.  Sixteen frames are read at a time: one after
// another each waits for memory (64 lanes x 262144 frames, 3 % of them triggers: 11 -> 9 us).
__global__ void latch_last_kernel(const float *__restrict__ cond, int cond_mode, int64_t T, int W, int NC,
                                  int *__restrict__ last, int *__restrict__ span, int NP) {
  dgc_after_previous();
  const int e = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
  if (e >= W) return;
  if (c < NP) span[(size_t)c * W + e] = 0;     // for latch_seg_kernel
  const int64_t n0 = (int64_t)c * LATCH_CHUNK, n1 = min(n0 + (int64_t)LATCH_CHUNK, T);
  constexpr int G = 16;
  static_assert(LATCH_CHUNK % G == 0, "whole groups");
  const int64_t stride = cond_mode == 1 ? 1 : W;
  const float *p = cond + (cond_mode == 1 ? n0 : n0 * W + e);
  const int cnt = (int)(n1 - n0);
  int found = -1;
  for (int g = (cnt - 1) / G * G; g >= 0 && found < 0; g -= G) {     // frames g .. g + 15 of the chunk
    float v[G], most = 0.0f;
    const float *q = p + g * stride;
#pragma unroll
    for (int j = 0; j < G; ++j, q += stride) v[j] = g + j < cnt ? *q : 0.0f;
#pragma unroll
    for (int j = 0; j < G; ++j) most = fmaxf(most, v[j]);
    if (most > 0.0f) {
#pragma unroll
      for (int j = 0; j < G; ++j)
        if (v[j] > 0.0f) found = g + j;
    }
  }
  last[(size_t)c * W + e] = found;
}

// Exclusive "most recent trigger" over chunks in two coalesced steps (threads run along the lanes):
//   segments of LATCH_SEG chunks: place of the last trigger inside each segment, chunk * LATCH_CHUNK + offset + 1 or 0 for
//   none; spans of LATCH_SPAN segments: the latest of theirs;
//   each (segment, lane) thread then looks back for the last one with a trigger, eight at a time, through the segments of
//   its span (mostly the one before it; a walk of one thread per lane over all of them was a launch of 9 us), then
//   through the spans, and walks its chunks: last[c][e] becomes the offset and src_chunk[c][e] the chunk of the most
//   recent trigger BEFORE chunk c (chunk -1: none yet, the state cell holds the value).  (Through the segments alone, a
//   trigger in 10 000 frames took 1025 us for 256 lanes x 2 M frames against 955 for that walk, now 855.)
constexpr int LATCH_SEG = 32, LATCH_SPAN = 32;

__global__ void latch_seg_kernel(const int *__restrict__ last, int W, int NC, int *__restrict__ seg, int *__restrict__ span) {
  dgc_after_previous();
  const int e = blockIdx.x * blockDim.x + threadIdx.x, sgm = blockIdx.y;
  if (e >= W) return;
  const int c0 = sgm * LATCH_SEG, c1 = min(c0 + LATCH_SEG, NC);
  int at = 0;
#pragma unroll 8
  for (int c = c0; c < c1; ++c) {
    const int v = last[(size_t)c * W + e];
    if (v >= 0) at = c * LATCH_CHUNK + v + 1;
  }
  seg[(size_t)sgm * W + e] = at;
  if (at) atomicMax(span + (size_t)(sgm / LATCH_SPAN) * W + e, at);
}

__global__ void latch_carry_kernel(int *last, int *src_chunk, const int *__restrict__ seg, const int *__restrict__ span, int W,
                                   int NC) {
  dgc_after_previous();
  const int e = blockIdx.x * blockDim.x + threadIdx.x, sgm = blockIdx.y;
  if (e >= W) return;
  const int c0 = sgm * LATCH_SEG, c1 = min(c0 + LATCH_SEG, NC);
  // the latest of rows first - 1, first - 2, .. end that is not 0
  auto look_back = [&](const int *__restrict__ rows, int first, int end) {
    constexpr int BACK = 8;
    int at = 0;
    for (int s = first - 1; s >= end && !at; s -= BACK) {
      int v[BACK];
#pragma unroll
      for (int j = 0; j < BACK; ++j) v[j] = rows[(size_t)max(s - j, end) * W + e];
#pragma unroll
      for (int j = 0; j < BACK; ++j) at = max(at, v[j]);      // places grow with the row
    }
    return at;
  };
  const int mine = sgm / LATCH_SPAN;
  int at = look_back(seg, sgm, mine * LATCH_SPAN);
  if (!at) at = look_back(span, mine, 0);
  int run = at ? (at - 1) / LATCH_CHUNK : -1, run_off = at ? (at - 1) % LATCH_CHUNK : 0;
#pragma unroll 8
  for (int c = c0; c < c1; ++c) {
    const int here = last[(size_t)c * W + e];
    src_chunk[(size_t)c * W + e] = run;
    last[(size_t)c * W + e] = run_off;
    if (here >= 0) {
      run = c;
      run_off = here;
    }
  }
}

__global__ void latch_out_kernel(const float *__restrict__ value, const float *__restrict__ cond, int cond_mode,
                                 int64_t T, int W, int NC, const int *__restrict__ src_off,
                                 const int *__restrict__ src_chunk, const float *__restrict__ state,
                                 float *__restrict__ y) {
  dgc_after_previous();
  const int e = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
  if (e >= W) return;
  const int sc = src_chunk[(size_t)c * W + e];
  float held = sc >= 0 ? value[((int64_t)sc * LATCH_CHUNK + src_off[(size_t)c * W + e]) * W + e]
                       : (state ? state[e] : 0.0f);
  const int64_t n0 = (int64_t)c * LATCH_CHUNK, n1 = min(n0 + (int64_t)LATCH_CHUNK, T);
  // groups of sixteen frames: all loads of a group are issued before the dependent selects and stores
  constexpr int G = 16;
  for (int64_t n = n0; n < n1; n += G) {
    float v[G], c[G];
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const int64_t m = min(n + j, n1 - 1);
      v[j] = __ldcs(value + m * W + e);
      c[j] = cond_at(cond, cond_mode, m, e, W);
    }
#pragma unroll
    for (int j = 0; j < G; ++j)
      if (n + j < n1) {
        if (c[j] > 0.0f) held = v[j];
        __stcs(y + (n + j) * W + e, held);
      }
  }
}

// The output pass with FOUR lanes per thread (W a multiple of 4): a warp reads 512 contiguous bytes of a frame, the
// block = (W / 4 lane groups) x (chunks) covers whole rows, results leave as 128-bit streaming stores.
// Bound by the loads in flight of the few threads that a chunk of 128 frames leaves: SHARED, one condition per frame, keeps
// sixteen frames of values on their way.  262144 frames of 64 lanes: 30 us with eight, 22.6 with sixteen.
template <bool SHARED>
__global__ void __launch_bounds__(256)
latch_out4_kernel(const float *__restrict__ value, const float *__restrict__ cond, int64_t T, int W, int NC,
                  const int *__restrict__ src_off, const int *__restrict__ src_chunk, const float *__restrict__ state,
                  float *__restrict__ y) {
  dgc_after_previous();
  const int e = (blockIdx.x * blockDim.x + threadIdx.x) * 4, c = blockIdx.y * blockDim.y + threadIdx.y;
  if (e >= W || c >= NC) return;
  float held[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int sc = src_chunk[(size_t)c * W + e + k];
    held[k] = sc >= 0 ? value[((int64_t)sc * LATCH_CHUNK + src_off[(size_t)c * W + e + k]) * W + e + k]
                      : (state ? state[e + k] : 0.0f);
  }
  const int64_t n0 = (int64_t)c * LATCH_CHUNK, n1 = min(n0 + (int64_t)LATCH_CHUNK, T);
  constexpr int G = SHARED ? 16 : 8;
  for (int64_t n = n0; n < n1; n += G) {
    float4 v[G], cc[SHARED ? 1 : G];
    float shared_cond[SHARED ? G : 1];
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const int64_t m = min(n + j, n1 - 1);
      v[j] = __ldcs(reinterpret_cast<const float4 *>(value + m * W + e));
      if constexpr (SHARED) shared_cond[j] = cond[m];
      else cc[j] = __ldcs(reinterpret_cast<const float4 *>(cond + m * W + e));
    }
#pragma unroll
    for (int j = 0; j < G; ++j)
      if (n + j < n1) {
        float4 c4;
        if constexpr (SHARED) c4 = make_float4(shared_cond[j], shared_cond[j], shared_cond[j], shared_cond[j]);
        else c4 = cc[j];
        if (c4.x > 0.0f) held[0] = v[j].x;
        if (c4.y > 0.0f) held[1] = v[j].y;
        if (c4.z > 0.0f) held[2] = v[j].z;
        if (c4.w > 0.0f) held[3] = v[j].w;
        __stcs(reinterpret_cast<float4 *>(y + (n + j) * W + e), make_float4(held[0], held[1], held[2], held[3]));
      }
  }
}

__global__ void latch_state_kernel(const float *__restrict__ y, int64_t T, int W, float *__restrict__ state) {
  dgc_after_previous();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < W) state[e] = y[(T - 1) * W + e];
}

// ---- compressor -------------------------------------------------------------------------------------------------
struct CompCoef {
  float ratio, threshold, inv_knee, att, rel, knee_start, knee_end, hard_ratio, thr_minus_start;
  bool forgets;   // nothing of the smoother's state is left after a tile
};

// 20 log10 of max(|a|, 1e-5): |a| = m 2^e with m in [sqrt(1/2), sqrt(2)), 20 log10(1 + f) = f p(f), f = m - 1, with p a
// least-squares fit of degree 8 reweighted towards equal relative error (at most 2.15 units in the last place of the result from
// 1e-5 to 32, at 0.986; 20 times a correctly rounded logarithm has more than that).  Branch-free, 17 instructions; the library call and the knee's divisions took 65 us
// of the kernel at 64 x 262144 samples.
__device__ __forceinline__ float amp2db(float a) {
  const float x = fmaxf(fabsf(a), 0.00001f);
  const int bits = __float_as_int(x), e = (bits - 0x3f3504f3) >> 23;
  const float f = __int_as_float(bits - (e << 23)) - 1.0f;
  float p = 0.75761503f;
  p = fmaf(p, f, -1.247889f);
  p = fmaf(p, f, 1.2987375f);
  p = fmaf(p, f, -1.4385911f);
  p = fmaf(p, f, 1.7334285f);
  p = fmaf(p, f, -2.1716526f);
  p = fmaf(p, f, 2.8953705f);
  p = fmaf(p, f, -4.3429437f);
  p = fmaf(p, f, 8.6858892f);
  const float db = fmaf((float)e, 6.0205999f, f * p);
  return x > 3.402823466e38f ? x : db;         // an infinite sample stays one
}

// The knee's slope 1 - 1 / r as (r - 1) / r, which loses no digits where r is close to 1.
__device__ __forceinline__ float gain_reduction(const CompCoef &c, float det_db) {
  // within 1e30 of zero: a limiter's ratio may be infinite, and the quotient is zero where its denominator is above 2^126
  const float pos = (det_db - c.knee_start) * c.inv_knee, rm1 = fminf(fmaxf(pos * (c.ratio - 1.0f), -1e30f), 1e30f);
  const float over = det_db - (c.knee_start + pos * c.thr_minus_start);
  const float soft = over * __fdividef(rm1, 1.0f + rm1);
  const float hard = (det_db - c.threshold) * c.hard_ratio;
  return det_db <= c.knee_start ? 0.0f : (det_db >= c.knee_end ? hard : soft);
}

// The attack / release smoother s <- c s + (1 - c) g, c = attack where g > s and release elsewhere, is the one recurrence
// of the op.  Its step is monotone and piecewise linear in s, so the states that enter the threads' runs of P samples
// are found by Newton's method on all of them at once: every thread walks its run from its present guess, which gives
// the run's end as an affine map A s + B of the state it started from (the branches held fixed), a scan of those maps
// over the block gives the next guesses, and when no guess moves by more than rounding the walk from them IS the
// recurrence.  After k rounds the first k runs are exact whatever the input; programme material needs 5 to 9 rounds, a
// square-wave level with a 1 s release 34.  The branch bits differ from the serial order's only where g = s within
// rounding, where both branches give the same value.
//
// One launch does the op: a block takes a tile of 512 P samples of one voice, in ticket order, tiles of all voices
// side by side: level detection (logarithm, knee) from coalesced loads into shared memory, the state its predecessor
// handed on, the smoother, y = sign(x) max(|x|, 1e-5) 10^(-s / 20) with coalesced stores.  x is read twice, the second
// time from L2.  Bound: instruction issue (about 20 per sample for the level and the gain, 10 per sample and round).
// 64 voices x 262144 samples: 123 us, 3290 us for a warp per voice that walked its samples one by one (3420 us with the
// two passes around it); without the rounds 57 us, of which 20 are HBM's.
//
// Where the level stands still the state ends up within rounding of it, the branch is decided by the last bit and a round
// settles one run.  After rounds that took about as long as that, one thread walks the tile in order: 1 x 16384 samples of
// a constant level, 50 ms release, 215 us (rounds alone 385, a warp per voice that walks its samples 222); 1 x 4096, 3 s
// release, 65 us (108 and 69).
constexpr int COMP_THREADS = 512;

struct Affine {
  float a, b;
};
// later o earlier; the factor is kept off zero so that an infinite state stays one instead of turning 0 x inf
__device__ __forceinline__ Affine affine_after(Affine later, Affine earlier) {
  return {fmaxf(later.a * earlier.a, 1.17549435e-38f), fmaf(later.a, earlier.b, later.b)};
}

template <int P>
__global__ void __launch_bounds__(COMP_THREADS, 2)
compressor_kernel(const float *__restrict__ x, const float *__restrict__ det, int B, int64_t T, int NT, CompCoef c,
                  float *state, float *__restrict__ y, unsigned long long *__restrict__ chain, int32_t *status) {
  dgc_after_previous();
  constexpr int TILE = COMP_THREADS * P, WARPS = COMP_THREADS / 32;
  extern __shared__ float gs[];                // TILE values, one pad float after every P: a thread's run is conflict-free
  __shared__ Affine warp_map[2][WARPS];
  __shared__ uint32_t sh_index;
  __shared__ float sh_state, entry[COMP_THREADS + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) sh_index = dgchain::take_ticket(chain);
  __syncthreads();
  const uint32_t index = sh_index;
  if (index >= (uint32_t)B * (uint32_t)NT) return;   // given up, or another launch has taken tickets of this one
  const int tile = (int)(index / (uint32_t)B), b = (int)(index - (uint32_t)tile * B);
  const int64_t n0 = (int64_t)tile * TILE;
  const int len = (int)min((int64_t)TILE, T - n0);
  const float *xt = x + (size_t)b * T + n0, *dt = det + (size_t)b * T + n0;
  float *yt = y + (size_t)b * T + n0;
  unsigned long long *cell = chain + 1 + 2 * ((size_t)b * NT + tile);   // end value, infinite state
  float g[P];
#pragma unroll
  for (int j = 0; j < P; ++j) {                // all loads of the tile in flight before the first is used
    const int i = j * COMP_THREADS + tid;
    g[j] = i < len ? __ldg(dt + i) : 0.0f;
  }
#pragma unroll
  for (int j = 0; j < P; ++j) {
    const int i = j * COMP_THREADS + tid;
    gs[i + i / P] = gain_reduction(c, amp2db(g[j]));
  }
  __syncthreads();
  const int cnt = max(0, min(P, len - tid * P));
#pragma unroll
  for (int j = 0; j < P; ++j) g[j] = j < cnt ? gs[tid * (P + 1) + j] : 0.0f;
  const float att = c.att, rel = c.rel, one_m_att = 1.0f - att, one_m_rel = 1.0f - rel;

  float s_in = 0.0f, guess = 0.0f, walked = 0.0f;
  Affine own = {1.0f, 0.0f};                   // this run's map and its end, walked from `walked`
  float end = 0.0f;
  bool stale = true;
  const bool whole = len == TILE;
  const int max_rounds = max(9, len / (P == 8 ? 256 : 512));   // about as long as the walk in order that follows them
  auto walk = [&](auto all) {
    float s = guess;
    own = {1.0f, 0.0f};
#pragma unroll
    for (int j = 0; j < P; ++j)
      if (decltype(all)::value || j < cnt) {
        const bool up = g[j] > s;
        const float k = up ? att : rel, d = g[j] * (up ? one_m_att : one_m_rel);
        s = fmaf(k, s, d);
        own.b = fmaf(k, own.b, d);
        own.a *= k;
      }
    end = s;
  };
  auto smoothed = [&](float s, float gn) {
    const float a_s = fmaf(att, s, gn * one_m_att), r_s = fmaf(rel, s, gn * one_m_rel);
    return gn > s ? a_s : r_s;
  };
  // A guess that moves by no more than rounding stands; so does an infinite one, and one that is no number.
  auto moves = [&] { return !(guess == walked || fabsf(guess - walked) <= 5e-7f * fabsf(guess) || (guess != guess && walked != walked)); };
  // The guesses come from the state at rest first: when the state that enters arrives only the runs it still reaches are
  // wrong.  And if nothing of a state is left after a tile (c^TILE below 2^-44, whatever branch is taken), the end value
  // found from rest goes out before the tile's own state is there: no work chained along time.  What a tile never forgets,
  // a state that is infinite or no number, passes from tile to tile beside it (zero: there is none).  Every tile takes
  // the same steps whether its predecessor is done or not, so the result does not depend on the order in which blocks run.
  bool sent = false, passed = !c.forgets;
  for (int pass = tile == 0 ? 1 : 0; pass < 2; ++pass) {
    if (pass == 1) {
      if (tid == COMP_THREADS - 1) {
        float s0 = 0.0f;
        if (tile > 0) {
          const float e = guess == walked ? end : fmaf(own.a, guess - walked, end);
          sent = c.forgets && whole;
          if (sent) dgchain::publish(cell, e);
          s0 = dgchain::await(cell - 2, chain, status);
          if (c.forgets) {
            const float p = dgchain::await(cell - 1, chain, status);
            if (p != 0.0f) s0 = p;
            else if (sent && fabsf(e) <= 3.402823466e38f) {
              dgchain::publish(cell + 1, 0.0f);
              passed = true;
            }
          }
        } else if (state) {
          s0 = state[b];
        }
        sh_state = s0;
      }
      __syncthreads();
      s_in = sh_state;
      if (tile == 0) guess = s_in;
      else if (tid == 0) {
        guess = s_in;
        stale = stale || moves();
      }
    }
    for (int round = 0;; ++round) {
      if (__any_sync(0xffffffffu, stale)) {    // a warp whose guesses stand keeps its maps
        walked = guess;
        if (whole) walk(std::true_type());     // most tiles: no count to test at every sample
        else walk(std::false_type());
      }
      Affine m = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const Affine e = {__shfl_up_sync(0xffffffffu, m.a, o), __shfl_up_sync(0xffffffffu, m.b, o)};
        if (lane >= o) m = affine_after(m, e);
      }
      if (lane == 31) warp_map[round & 1][warp] = m;
      __syncthreads();
      // every warp composes the maps of the warps before it
      Affine w = lane < warp ? warp_map[round & 1][lane] : Affine{1.0f, 0.0f};
#pragma unroll
      for (int o = 1; o < WARPS; o <<= 1) {
        const Affine e = {__shfl_up_sync(0xffffffffu, w.a, o), __shfl_up_sync(0xffffffffu, w.b, o)};
        if (lane >= o) w = affine_after(w, e);
      }
      w = {__shfl_sync(0xffffffffu, w.a, WARPS - 1), __shfl_sync(0xffffffffu, w.b, WARPS - 1)};
      const float warp_in = fmaf(w.a, s_in, w.b);
      guess = __shfl_up_sync(0xffffffffu, fmaf(m.a, warp_in, m.b), 1);
      if (lane == 0) guess = warp == 0 ? s_in : warp_in;
      stale = moves();
      if (!__syncthreads_or(stale)) break;
      if (round == max_rounds) {               // one thread walks the tile in order, its loads sixteen samples ahead
        stale = true;
        if (tid == 0) {
          constexpr int G = 16;
          float s = s_in, now[G], next[G];
          auto load = [&](int i0, float (&v)[G]) {
#pragma unroll
            for (int j = 0; j < G; ++j) v[j] = gs[i0 + j + (i0 + j) / P];
          };
          load(0, now);
          for (int i0 = 0; i0 < len; i0 += G) {
            load(min(i0 + G, TILE - G), next);
#pragma unroll
            for (int j = 0; j < G; ++j) {
              if ((i0 + j) % P == 0) entry[(i0 + j) / P] = s;
              s = smoothed(s, now[j]);
            }
#pragma unroll
            for (int j = 0; j < G; ++j) now[j] = next[j];
          }
          entry[COMP_THREADS] = s;             // read where the tile is whole
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < P; ++j) g[j] = j < cnt ? gs[tid * (P + 1) + j] : 0.0f;   // not kept in registers over the walk
        guess = walked = entry[tid];
        end = entry[tid + 1];
        break;                                 // (stale stays set: the next pass walks every run anew)
      }
    }
  }
  float s = guess;
#pragma unroll
  for (int j = 0; j < P; ++j)
    if (j < cnt) gs[tid * (P + 1) + j] = s = smoothed(s, g[j]);
  if (cnt > 0 && tid * P + cnt == len) {       // the thread of the tile's last sample
    if (tile == NT - 1) {
      if (state) state[b] = s;                 // the first tile has read it: what it published has led to this one
    } else {
      if (!sent) dgchain::publish(cell, s);
      if (!passed) dgchain::publish(cell + 1, fabsf(s) <= 3.402823466e38f ? 0.0f : s);
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < P; ++j) {
    const int i = j * COMP_THREADS + tid;
    g[j] = i < len ? __ldcs(xt + i) : 0.0f;
  }
#pragma unroll
  for (int j = 0; j < P; ++j) {
    const int i = j * COMP_THREADS + tid;
    if (i < len) {
      const float v = g[j], a = fmaxf(fabsf(v), 0.00001f) * exp10f(gs[i + i / P] * -0.05f);
      __stcs(yt + i, v > 0.0f ? a : (v < 0.0f ? -a : 0.0f));
    }
  }
}

// ---- phase vocoder ----------------------------------------------------------------------------------------------
// Emit+PhaseVocoder.swift:46-53
__device__ __forceinline__ float principal_arg(float v) {
  const float tau = 6.28318530717958647692f, half = 3.14159265358979323846f;
  const float w = v - tau * roundf(v / tau);
  const float wh = w > half ? w - tau : w;
  return w < -half ? wh + tau : wh;
}

// The same for the running phase of the synthesis, where a step's latency counts and a multiple of tau more or less is the
// same phase: turns counted by a multiplication and rounded to the nearest even by an addition (below 2^22 turns; a single-
// precision phase beyond has no fraction left).  A count that its rounding makes one too many or too few leaves the phase just
// outside half a turn; it is folded at every step, so that a stream cut in two calls goes on with what one call has.
__device__ __forceinline__ float wrapped(float v) {
  const float tau = 6.28318530717958647692f, half = 3.14159265358979323846f, big = 12582912.0f;
  const float w = fmaf(-tau, fmaf(v, 0.15915494309189533577f, big) - big, v);
  const float folded = w - copysignf(tau, w);
  return fabsf(w) > half ? folded : w;
}

// Sine and cosine of a wrapped phase, each to 1.5e-7: folded about a quarter turn, then both polynomials in x^2 (minimax on that
// range, 1e-11 and 2e-10) as the halves of packed multiply-adds: 16 instructions, the library's pair takes three times as many.
// A phase that is not wrapped (a state handed in, nothing finite) goes to the library.
__device__ __noinline__ float2 sincos_any(float p) {
  float2 r;
  sincosf(p, &r.y, &r.x);
  return r;
}
__device__ __forceinline__ void sincos_wrapped(float p, float &s, float &c) {
  if (!(fabsf(p) <= 3.2f)) {
    const float2 r = sincos_any(p);
    s = r.y;
    c = r.x;
    return;
  }
  const bool far = fabsf(p) > 1.57079632679489661923f;
  const float x = far ? (copysignf(3.1415927410125732422f, p) - p) - copysignf(8.7422776573475857731e-8f, p) : p;
  const float z = x * x;
  const float2 zz = make_float2(z, z);
  float2 q = make_float2(-2.3794711816e-8f, -2.6051493821e-7f);
  q = __ffma2_rn(q, zz, make_float2(2.7518855533e-6f, 2.4760161284e-5f));
  q = __ffma2_rn(q, zz, make_float2(-1.9840702860e-4f, -1.3888361399e-3f));
  q = __ffma2_rn(q, zz, make_float2(8.3333292644e-3f, 4.1666636258e-2f));
  q = __ffma2_rn(q, zz, make_float2(-1.6666666541e-1f, -4.9999999359e-1f));
  q = __ffma2_rn(q, zz, make_float2(1.0f, 1.0f));
  s = q.x * x;
  c = far ? -q.y : q.y;
}

__device__ __forceinline__ float mixf(float a, float b, float t) { return fmaf(b, t, a * (1.0f - t)); }

// Analysis (Emit+PhaseVocoder.swift:57-71), parallel over (voice, bin, runs of hops): the "previous analysis phase" of hop h
// is the phase of hop h - 1 of the INPUT (the state cell only for the first hop of the call), so nothing here is a
// recurrence.  A thread takes PV_RUN hops of a bin and so evaluates one arc tangent per element (and one for the hop before
// the run), four hops in flight (eight at once outgrew the instruction cache): 33 us, 35 with eight, 70 with two arc tangents per
// element.  Magnitude and frequency go out side by side: the synthesis gathers both at the same places.
constexpr int PV_RUN = 8, PV_AHEAD = 4;
__global__ void __launch_bounds__(128)
pv_analysis_kernel(const float *__restrict__ re, const float *__restrict__ im, int64_t H, int N, float omega_scale,
                   const float *__restrict__ state, float2 *__restrict__ mag_omega) {
  dgc_after_previous();
  const int i = blockIdx.y * blockDim.x + threadIdx.x, v = blockIdx.z;
  const int64_t h0 = (int64_t)blockIdx.x * PV_RUN;
  if (i >= N) return;
  const size_t at = ((size_t)v * H + h0) * N + i;
  const int cnt = (int)min((int64_t)PV_RUN, H - h0);
  const float *pr = re + at, *pq = im + at;
  float2 *out = mag_omega + at;
  float prev = h0 > 0 ? atan2f(im[at - N], re[at - N]) : (state ? state[(size_t)v * (2 * N + 1) + i] : 0.0f);
  const float target = (float)i * omega_scale;
#pragma unroll 1
  for (int j0 = 0; j0 < cnt; j0 += PV_AHEAD) {
    float r[PV_AHEAD], q[PV_AHEAD];
#pragma unroll
    for (int j = 0; j < PV_AHEAD; ++j) {
      const bool in = j0 + j < cnt;
      r[j] = in ? pr[(ptrdiff_t)j * N] : 0.0f;
      q[j] = in ? pq[(ptrdiff_t)j * N] : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < PV_AHEAD; ++j)
      if (j0 + j < cnt) {
        const float phase = atan2f(q[j], r[j]);
        out[(ptrdiff_t)j * N] = make_float2(sqrtf(r[j] * r[j] + q[j] * q[j]), target + principal_arg(phase - prev - target));
        prev = phase;
      }
    pr += (size_t)PV_AHEAD * N;
    pq += (size_t)PV_AHEAD * N;
    out += (size_t)PV_AHEAD * N;
  }
}

// Resynthesis (Emit+PhaseVocoder.swift:73-108): the synthesis phase of an output bin is the one value carried from hop to
// hop, one addition and one wrap.  Everything else about a hop -- where its bin comes from, the gathered pairs of
// (magnitude, frequency), sine and cosine -- is independent of it.  A block takes 32 bins of a voice, tile after tile of 32
// hops; eight warps share a tile's hops, four each.  While a ninth warp adds up one tile's frequencies in hop order, the eight
// leave the next tile's in shared memory, turn the tile before into spectra and send for the one after the next: one barrier a
// tile, three tiles of shared memory.  Bound by issue (a division, a gather and a sine and cosine per element).  8 voices x 469
// hops x 2048 bins: 522 us for a thread per bin that did everything in hop order, 82 with the library's sine and one of the
// eight warps adding between two barriers, 71 with the sine above, 63 like this.
// ratio_mode 0: one value, 1: [H], 2: [V][H].
constexpr int PV_BINS = 32, PV_WARPS = 8, PV_PER = 4, PV_TILE = PV_WARPS * PV_PER, PV_THREADS = PV_BINS * (PV_WARPS + 1);
__global__ void __launch_bounds__(PV_THREADS, 4)
pv_synthesis_kernel(const float *__restrict__ re, const float *__restrict__ im, const float2 *__restrict__ mag_omega,
                    const float *__restrict__ ratio, int ratio_mode, int64_t H, int N, float *__restrict__ state,
                    float *__restrict__ out_re, float *__restrict__ out_im) {
  dgc_after_previous();
  __shared__ float phase[3][PV_TILE][PV_BINS];      // a tile's unscaled frequencies, then, in place, its phases
  __shared__ float ratios[3][PV_TILE];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, v = blockIdx.y;
  const int k = blockIdx.x * PV_BINS + lane;
  const bool live = k < N;
  float *st = state ? state + (size_t)v * (2 * N + 1) : nullptr;
  const bool started = st ? st[2 * N] != 0.0f : false;
  const size_t base = (size_t)v * H * N;
  const int tiles = (int)((H + PV_TILE - 1) / PV_TILE);
  if (warp == PV_WARPS) {                            // the one that adds
    float synth = st && live ? st[N + k] : 0.0f;
    __syncthreads();
    for (int t = 0, slot = 0; t <= tiles; ++t, slot = slot == 2 ? 0 : slot + 1) {
      if (t < tiles) {
        const int cnt = (int)min((int64_t)PV_TILE, H - (int64_t)t * PV_TILE);
#pragma unroll 8
        for (int j = 0; j < cnt; ++j) {
          const float om = phase[slot][j][lane];
          synth = t + j == 0 && !started ? om : wrapped(fmaf(om, ratios[slot][j], synth));
          phase[slot][j][lane] = synth;
        }
      }
      __syncthreads();
    }
    if (st && live) {
      const size_t last = base + (size_t)(H - 1) * N + k;
      // the "started" flag is shared by all bins of a voice and other blocks may still have to read it: a launch of
      // its own sets it afterwards
      st[N + k] = synth;
      st[k] = atan2f(im[last], re[last]);
    }
    return;
  }
  const float nm1 = (float)(N - 1), kf = (float)k;
  const int w0 = warp * PV_PER;                      // this thread's first hop of a tile
  const float *ratio_v = ratio_mode == 2 ? ratio + (size_t)v * H : ratio;
  const float2 *rows = mag_omega + base + (size_t)w0 * N;        // of the tile that is fetched
  float *o_re = out_re + base + (size_t)w0 * N + k, *o_im = out_im + base + (size_t)w0 * N + k;   // of the tile that goes out
  float mag[2][PV_PER], frac[PV_PER], r[PV_PER];     // magnitudes of the tile that is added up and of the next one
  float2 lo[PV_PER], hi[PV_PER];
  unsigned in_range = 0;
  // this thread's hops of tile t: where their bin comes from, and the loads of the two pairs there
  auto fetch = [&](int t) {
    in_range = 0;
    const int64_t h0 = (int64_t)t * PV_TILE;
    const int last = (int)min((int64_t)PV_TILE, H - h0) - 1 - w0;   // the last hop of them there is (below zero: none)
#pragma unroll
    for (int j = 0; j < PV_PER; ++j) {
      const int jj = min(j, last);                   // a hop past the end reads the last one's
      r[j] = fmaxf(ratio_mode == 0 ? ratio[0] : ratio_v[h0 + w0 + jj], 1e-4f);
      const float src = kf / r[j];
      const bool in = src <= nm1;
      if (in) in_range |= 1u << j;
      const float srcc = in ? src : nm1, fl = floorf(srcc);
      frac[j] = srcc - fl;
      const int i0 = (int)fl, i1 = i0 < N - 1 ? i0 + 1 : i0;
      const float2 *row = rows + (ptrdiff_t)jj * N;
      lo[j] = __ldg(row + i0);
      hi[j] = __ldg(row + i1);
      if (t == 0 && w0 + j == 0 && !started) {
        // first hop of the stream: start from the interpolated analysis phase of this hop
        const float p0 = atan2f(im[base + i0], re[base + i0]), p1 = atan2f(im[base + i1], re[base + i1]);
        phase[0][0][lane] = principal_arg(mixf(p0, p1, frac[j]));
      }
    }
    rows += (size_t)PV_TILE * N;
  };
  // what was fetched: the magnitudes kept, the frequencies for the one that adds
  auto leave = [&](int t, int slot) {
#pragma unroll
    for (int j = 0; j < PV_PER; ++j) {
      mag[0][j] = mag[1][j];
      mag[1][j] = in_range & (1u << j) ? mixf(lo[j].x, hi[j].x, frac[j]) : 0.0f;
      if (t > 0 || w0 + j > 0 || started) phase[slot][w0 + j][lane] = mixf(lo[j].y, hi[j].y, frac[j]);
      if (lane == 0) ratios[slot][w0 + j] = r[j];
    }
  };
  if (live) {
    fetch(0);
    leave(0, 0);
    if (tiles > 1) fetch(1);
  }
  __syncthreads();
  for (int t = 0, slot = 0; t <= tiles; ++t, slot = slot == 2 ? 0 : slot + 1) {   // tile t is added up
    if (live) {
      float before[PV_PER];
#pragma unroll
      for (int j = 0; j < PV_PER; ++j) before[j] = mag[0][j];
      if (t + 1 < tiles) {
        leave(t + 1, slot == 2 ? 0 : slot + 1);
        if (t + 2 < tiles) fetch(t + 2);
      } else {
#pragma unroll
        for (int j = 0; j < PV_PER; ++j) mag[0][j] = mag[1][j];
      }
      if (t > 0) {
        const int cnt = (int)min((int64_t)PV_PER, H - (int64_t)(t - 1) * PV_TILE - w0);
#pragma unroll
        for (int j = 0; j < PV_PER; ++j)
          if (j < cnt) {
            float sn, cs;
            sincos_wrapped(phase[slot == 0 ? 2 : slot - 1][w0 + j][lane], sn, cs);
            o_re[(ptrdiff_t)j * N] = before[j] * cs;
            o_im[(ptrdiff_t)j * N] = before[j] * sn;
          }
        o_re += (size_t)PV_TILE * N;
        o_im += (size_t)PV_TILE * N;
      }
    }
    __syncthreads();
  }
}

__global__ void pv_mark_started_kernel(float *state, int V, int N) {
  dgc_after_previous();
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < V) state[(size_t)v * (2 * N + 1) + 2 * N] = 1.0f;
}

}  // namespace

// ---------------------------------------------------------------------------------------------------------------
DGC_EXPORT int32_t dgc_delay_line(dgc_ctx *ctx, const float *x_dev, const float *delay_dev, int32_t delay_mode,
                                  int64_t T, int32_t lanes, int32_t max_delay, float *ring_dev, float *head_dev,
                                  float *y_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, x_dev && delay_dev && y_dev, "null pointer");
  DGC_REQUIRE(ctx, T > 0 && lanes > 0, "size out of range");
  DGC_REQUIRE(ctx, max_delay > 1 && max_delay <= (1 << 24), "max_delay must be in 2..2^24 (the head is a float cell)");
  DGC_REQUIRE(ctx, delay_mode >= 0 && delay_mode <= 3, "delay_mode must be 0 (one value), 1 ([T]), 2 ([T][lanes]) or 3 ([lanes])");
  DGC_REQUIRE(ctx, (ring_dev == nullptr) == (head_dev == nullptr), "ring and head must be given together");
  DGC_REQUIRE(ctx, x_dev != y_dev, "in-place operation is not supported");
  DGC_REQUIRE(ctx, T * lanes / 256 < 0x7fffffffLL, "T * lanes too large");
  launch_frac_delay<false>(ctx->stream, x_dev, delay_dev, delay_mode, 0, T, lanes, max_delay, (float)(max_delay - 1),
                           ring_dev, head_dev, y_dev);
  DGC_LAUNCHED(ctx, "delay_line");
  if (ring_dev) {
    dgc_launch(ring_update_kernel<false>, dgc_div_up((int64_t)lanes * max_delay, 256), 256, 0, ctx->stream, x_dev, T, lanes,
               max_delay, ring_dev, head_dev);
    DGC_LAUNCHED(ctx, "delay_line_ring");
    dgc_launch(head_advance_kernel, 1, 1, 0, ctx->stream, head_dev, T, max_delay);
    DGC_LAUNCHED(ctx, "delay_line_head");
  }
  return DGC_OK;
}

DGC_EXPORT int32_t dgc_spectrum_delay(dgc_ctx *ctx, const float *spec_dev, const float *delay_dev, int64_t H,
                                      int32_t N, int32_t hops, float *ring_dev, float *row_dev, float *out_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, spec_dev && out_dev, "null pointer");
  DGC_REQUIRE(ctx, H > 0 && N > 0, "size out of range");
  DGC_REQUIRE(ctx, hops >= 1 && hops < (1 << 24), "hops must be in 1..2^24-1");
  DGC_REQUIRE(ctx, (ring_dev == nullptr) == (row_dev == nullptr), "ring and row must be given together");
  DGC_REQUIRE(ctx, spec_dev != out_dev, "in-place operation is not supported");
  DGC_REQUIRE(ctx, H * N / 256 < 0x7fffffffLL, "H * N too large");
  const int R = hops + 1;
  // fixed delay: the spectrum of exactly `hops` boundaries ago; modulated: per-hop delay in [0, hops]
  launch_frac_delay<true>(ctx->stream, spec_dev, delay_dev, delay_dev ? 1 : -1, hops, H, N, R, (float)hops, ring_dev,
                          row_dev, out_dev);
  DGC_LAUNCHED(ctx, "spectrum_delay");
  if (ring_dev) {
    dgc_launch(ring_update_kernel<true>, dgc_div_up((int64_t)N * R, 256), 256, 0, ctx->stream, spec_dev, H, N, R, ring_dev,
               row_dev);
    DGC_LAUNCHED(ctx, "spectrum_delay_ring");
    dgc_launch(head_advance_kernel, 1, 1, 0, ctx->stream, row_dev, H, R);
    DGC_LAUNCHED(ctx, "spectrum_delay_row");
  }
  return DGC_OK;
}

DGC_EXPORT uint64_t dgc_latch_scratch_floats(int64_t T, int32_t lanes) {
  if (T <= 0 || lanes <= 0) return 0;
  const uint64_t NC = (uint64_t)((T + LATCH_CHUNK - 1) / LATCH_CHUNK), NS = (NC + LATCH_SEG - 1) / LATCH_SEG;
  return (2 * NC + 2 * NS) * (uint64_t)lanes;
}

DGC_EXPORT int32_t dgc_latch(dgc_ctx *ctx, const float *value_dev, const float *cond_dev, int32_t cond_mode, int64_t T,
                             int32_t lanes, float *state_dev, float *scratch_dev, float *y_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, value_dev && cond_dev && y_dev, "null pointer");
  DGC_REQUIRE(ctx, T > 0 && lanes > 0, "size out of range");
  DGC_REQUIRE(ctx, cond_mode == 1 || cond_mode == 2, "cond_mode must be 1 ([T]) or 2 ([T][lanes])");
  const int64_t NC64 = (T + LATCH_CHUNK - 1) / LATCH_CHUNK;
  DGC_REQUIRE(ctx, NC64 <= 65535, "T too large");
  const int NC = (int)NC64;
  float *scr = scratch_dev ? scratch_dev : dgc_ctx_scratch(ctx, dgc_latch_scratch_floats(T, lanes));
  if (!scr) return DGC_ERR_OOM;
  int *last = reinterpret_cast<int *>(scr), *src_chunk = last + (size_t)NC * lanes;
  dim3 grid(dgc_div_up(lanes, 128), NC);
  const int NS = dgc_div_up(NC, LATCH_SEG), NP = dgc_div_up(NS, LATCH_SPAN);
  int *seg = src_chunk + (size_t)NC * lanes, *span = seg + (size_t)NS * lanes;
  dgc_launch(latch_last_kernel, grid, 128, 0, ctx->stream, cond_dev, cond_mode, T, lanes, NC, last, span, NP);
  DGC_LAUNCHED(ctx, "latch_last");
  dim3 sgrid(dgc_div_up(lanes, 128), NS);
  dgc_launch(latch_seg_kernel, sgrid, 128, 0, ctx->stream, last, lanes, NC, seg, span);
  DGC_LAUNCHED(ctx, "latch_segments");
  dgc_launch(latch_carry_kernel, sgrid, 128, 0, ctx->stream, last, src_chunk, seg, span, lanes, NC);
  DGC_LAUNCHED(ctx, "latch_carry");
  const bool quad = (lanes & 3) == 0 &&
                    ((((uintptr_t)value_dev) | ((uintptr_t)y_dev) | (cond_mode == 2 ? (uintptr_t)cond_dev : 0)) & 15) == 0;
  if (quad) {
    const int bx = lanes / 4 >= 64 ? 64 : lanes / 4, by = 256 / bx >= 1 ? (256 / bx > 8 ? 8 : 256 / bx) : 1;
    auto kern = cond_mode == 1 ? latch_out4_kernel<true> : latch_out4_kernel<false>;
    dgc_launch(kern, dim3(dgc_div_up(lanes / 4, bx), dgc_div_up(NC, by)), dim3(bx, by), 0, ctx->stream, value_dev, cond_dev, T,
               lanes, NC, last, src_chunk, state_dev, y_dev);
  } else {
    dgc_launch(latch_out_kernel, grid, 128, 0, ctx->stream, value_dev, cond_dev, cond_mode, T, lanes, NC, last, src_chunk,
               state_dev, y_dev);
  }
  DGC_LAUNCHED(ctx, "latch_out");
  if (state_dev) {
    dgc_launch(latch_state_kernel, dgc_div_up(lanes, 128), 128, 0, ctx->stream, y_dev, T, lanes, state_dev);
    DGC_LAUNCHED(ctx, "latch_state");
  }
  return DGC_OK;
}

DGC_EXPORT int32_t dgc_compressor(dgc_ctx *ctx, const dgc_compressor_params *p, const float *x_dev,
                                  const float *sidechain_dev, float *state_dev, float *y_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, p && x_dev && y_dev, "null pointer");
  DGC_REQUIRE(ctx, p->B > 0 && p->T > 0, "size out of range");
  DGC_REQUIRE(ctx, p->attack > 0.0f && p->release > 0.0f && p->sample_rate > 0.0f, "attack, release and sample_rate must be positive");
  CompCoef c;
  c.ratio = p->ratio;
  c.threshold = p->threshold;
  c.inv_knee = 1.0f / p->knee;
  // exp(log(0.01) / (time * sample_rate)), single precision as the reference graph evaluates it
  const float log001 = logf(0.01f);
  c.att = expf(log001 / (p->attack * p->sample_rate));
  c.rel = expf(log001 / (p->release * p->sample_rate));
  const float half = p->knee / 2.0f;
  c.knee_start = p->threshold - half;
  c.knee_end = p->threshold + half;
  c.hard_ratio = 1.0f - 1.0f / p->ratio;
  c.thr_minus_start = p->threshold - c.knee_start;
  DGC_REQUIRE(ctx, x_dev != y_dev && sidechain_dev != y_dev, "in-place operation is not supported");
  const int64_t n = (int64_t)p->B * p->T;
  DGC_REQUIRE(ctx, n / 256 < 0x7fffffffLL, "B * T too large");
  // 32 samples per thread: a long signal's tiles follow one another, so few and large ones; 8 where one small tile or two
  // hold the whole signal and its logarithms should spread over more than one SM
  const float *det = sidechain_dev ? sidechain_dev : x_dev;
  const int P = p->T <= 8192 ? 8 : 32, tile = COMP_THREADS * P;
  const int NT = dgc_div_up(p->T, tile), smem = (tile + COMP_THREADS) * (int)sizeof(float);
  c.forgets = powf(fmaxf(c.att, c.rel), (float)tile) < 5.7e-14f;
  const uint64_t blocks = (uint64_t)p->B * NT;
  DGC_REQUIRE(ctx, blocks <= 0x7fffffffull, "B * T too large");
  unsigned long long *chain = dgc_ctx_chain(ctx, 2 * blocks);
  if (!chain) return DGC_ERR_OOM;
  if (P == 8) {
    dgc_launch(compressor_kernel<8>, (unsigned)blocks, COMP_THREADS, smem, ctx->stream, x_dev, det, p->B, p->T, NT, c, state_dev,
               y_dev, chain, ctx->status_dev);
  } else {
    DGC_CUDA(ctx, cudaFuncSetAttribute(compressor_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    dgc_launch(compressor_kernel<32>, (unsigned)blocks, COMP_THREADS, smem, ctx->stream, x_dev, det, p->B, p->T, NT, c,
               state_dev, y_dev, chain, ctx->status_dev);
  }
  DGC_LAUNCHED(ctx, "compressor");
  return DGC_OK;
}

DGC_EXPORT uint64_t dgc_phase_vocoder_scratch_floats(int32_t V, int64_t H, int32_t N) {
  if (V <= 0 || H <= 0 || N <= 0) return 0;
  return 2ull * (uint64_t)V * (uint64_t)H * (uint64_t)N;
}

DGC_EXPORT int32_t dgc_phase_vocoder(dgc_ctx *ctx, const float *re_dev, const float *im_dev, const float *ratio_dev,
                                     int32_t ratio_mode, int32_t V, int64_t H, int32_t N, int32_t hop, float *state_dev,
                                     float *scratch_dev, float *out_re_dev, float *out_im_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, re_dev && im_dev && ratio_dev && out_re_dev && out_im_dev, "null pointer");
  DGC_REQUIRE(ctx, V > 0 && V <= 65535 && H > 0 && N > 0 && hop > 0, "size out of range");
  DGC_REQUIRE(ctx, ratio_mode >= 0 && ratio_mode <= 2, "ratio_mode must be 0 (one value), 1 ([H]) or 2 ([V][H])");
  DGC_REQUIRE(ctx, re_dev != out_re_dev && im_dev != out_im_dev, "in-place operation is not supported");
  const int64_t total = (int64_t)V * H * N;
  DGC_REQUIRE(ctx, total / 256 < 0x7fffffffLL, "V * H * N too large");
  const int64_t runs = (H + PV_RUN - 1) / PV_RUN;
  // pairs of floats: a caller's work space on an odd float is left for the context's own
  float *scr = scratch_dev && (((uintptr_t)scratch_dev) & 7) == 0 ? scratch_dev
                                                                   : dgc_ctx_scratch(ctx, dgc_phase_vocoder_scratch_floats(V, H, N));
  if (!scr) return DGC_ERR_OOM;
  float2 *mag_omega = reinterpret_cast<float2 *>(scr);
  const float omega_scale = 2.0f * 3.14159265358979323846f * (float)hop / (float)N;
  dgc_launch(pv_analysis_kernel, dim3((unsigned)runs, dgc_div_up(N, 128), V), 128, 0, ctx->stream, re_dev, im_dev, H, N,
             omega_scale, state_dev, mag_omega);
  DGC_LAUNCHED(ctx, "phase_vocoder_analysis");
  dgc_launch(pv_synthesis_kernel, dim3(dgc_div_up(N, PV_BINS), V), PV_THREADS, 0, ctx->stream, re_dev, im_dev, mag_omega,
             ratio_dev, ratio_mode, H, N, state_dev, out_re_dev, out_im_dev);
  DGC_LAUNCHED(ctx, "phase_vocoder_synthesis");
  if (state_dev) {
    dgc_launch(pv_mark_started_kernel, dgc_div_up(V, 128), 128, 0, ctx->stream, state_dev, V, N);
    DGC_LAUNCHED(ctx, "phase_vocoder_state");
  }
  return DGC_OK;
}
