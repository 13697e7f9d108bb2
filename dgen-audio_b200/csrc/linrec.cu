// Linear recurrences over time as chunked parallel scans: one-pole history feedback, the tensor
// biquad bank forward, and the reverse-time (BPTT) pass that yields coefficient gradients.
//
// The reference runs these per sample through history cells (Sources/DGen/Emit+State.swift:150-224,
// Sources/DGen/HigherOps.swift:401-570): one thread per lane, a serial loop over frames, and for
// BPTT a stored forward tape plus a reverse loop (Sources/DGen/Blocks/Emission/BPTTEmission.swift:471-518).
// Here time is cut into chunks; every (lane, chunk) runs the recurrence from a zero state, the
// chunk-to-chunk carry is an affine map (a power of the 2x2 transition matrix) resolved by a short
// scan, and a second sweep produces the output (forward) or the gradient sums (backward; by
// linearity the sums are corrected for the carried adjoint state without re-reading the signals).
#include <math.h>

#include <type_traits>

#include "chain.cuh"
#include "common.cuh"

namespace {

// ---------------------------------------------------------------------------------------------
// one-pole  y[n] = x[n] + a*y[n-1]
// ---------------------------------------------------------------------------------------------
// One launch: a block takes a tile of 2048 frames of one voice (ticket order, tiles of all voices side by side), runs it
// from rest, publishes its end value, sums the end values of the tiles before it -- decayed, in a fixed order, in double,
// as far back as a^(2048 j) is not yet nothing in single precision -- and writes the tile from that state.  Nothing waits
// for anything but end values, which need no wait themselves, so there is no chain along time, and x is read once: bound
// by HBM, short of it by the latency of a tile (load, scan, end value, store) over eight resident blocks.  64 x 262144
// frames: 40 us and 3 for clearing the cells, against 66 us for a pass for the end values, a serial carry and a second pass;
// 1 x 65536: one launch of 4 us, and 1, instead of three of 11.
// A state that is infinite or no number is never nothing: a tile that ends in one tags its cell, and the block that leaves
// last carries such a state to the end of its voice (a microsecond for the last block to be known; most calls have none).
// The sum is for filters that forget within OP_REACH tiles (|a| up to 0.9991).  Beyond, it grows with the memory, at last
// with the square of T, and three launches take over: 16 x 4 M frames 150 us for 0.9, 255 for 0.999, 365 for 0.9999 and 560
// for 1 as one launch, 227 as three; 64 x 262144: 55, 61, 58, 58 and 64.
constexpr int OP_THREADS = 128, OP_PER = 16, OP_TILE = OP_THREADS * OP_PER, OP_WARPS = OP_THREADS / 32;
constexpr int OP_BLOCKS = 8;    // resident per SM
constexpr int OP_REACH = 64;

// powers of the coefficient, evaluated in double on the host and rounded once
struct OnepolePowers {
  float a, r[7];          // a, and r^(2^i) with r = a^OP_PER
  double tile[6];         // A^(2^i) with A = a^OP_TILE
  int reach;              // tiles whose end values still matter: |A|^reach vanishes in single precision
};

OnepolePowers onepole_powers(float a) {
  OnepolePowers p;
  p.a = a;
  double r = 1.0;
  for (int i = 0; i < OP_PER; ++i) r *= (double)a;
  for (int i = 0; i < 7; ++i) {
    p.r[i] = (float)r;
    r *= r;
  }
  for (int i = 0; i < 6; ++i) {                      // r is now a^(OP_PER 2^7) = a^OP_TILE
    // kept finite: what grows beyond that is infinite in single precision, but silence times it stays silence
    p.tile[i] = r = fmin(r, 1e300);
    r *= r;
  }
  static_assert(OP_TILE == OP_PER << 7, "the powers double from a thread's run to a tile");
  const double lg = fabs(p.tile[0]) > 0.0 ? log2(fabs(p.tile[0])) : -1e30;
  p.reach = lg >= -1e-7 ? 0x7fffffff : (int)fmin(ceil(-160.0 / lg), 1e9);
  return p;
}

// A thread's run of sixteen frames is 64 contiguous bytes: four 128-bit accesses when it lies on a 16-byte boundary.
// REV: the scan's frame n is memory index T-1-n, the run is then read high to low.
template <bool REV>
__device__ __forceinline__ void onepole_load(const float *xb, int T, int n0, float *v) {
  const int m0 = REV ? T - n0 - OP_PER : n0;
  if (n0 + OP_PER <= T && ((uintptr_t)(xb + m0) & 15) == 0) {
#pragma unroll
    for (int q = 0; q < OP_PER / 4; ++q) {
      const float4 u = *(reinterpret_cast<const float4 *>(xb + m0) + q);
      const int k = REV ? OP_PER - 1 - 4 * q : 4 * q, d = REV ? -1 : 1;
      v[k] = u.x; v[k + d] = u.y; v[k + 2 * d] = u.z; v[k + 3 * d] = u.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < OP_PER; ++j) v[j] = (n0 + j < T) ? xb[REV ? T - 1 - (n0 + j) : n0 + j] : 0.0f;
  }
}

template <bool REV>
__device__ __forceinline__ void onepole_store(float *yb, int T, int n0, const float *v) {
  const int m0 = REV ? T - n0 - OP_PER : n0;
  if (n0 + OP_PER <= T && ((uintptr_t)(yb + m0) & 15) == 0) {
#pragma unroll
    for (int q = 0; q < OP_PER / 4; ++q) {
      const int k = REV ? OP_PER - 1 - 4 * q : 4 * q, d = REV ? -1 : 1;
      __stcs(reinterpret_cast<float4 *>(yb + m0) + q, make_float4(v[k], v[k + d], v[k + 2 * d], v[k + 3 * d]));
    }
  } else {
#pragma unroll
    for (int j = 0; j < OP_PER; ++j)
      if (n0 + j < T) yb[REV ? T - 1 - (n0 + j) : n0 + j] = v[j];
  }
}

// For the last block of a launch: the state that is infinite or no number at the end of a voice's first tagged tile, where
// the voice is finite after that.  (A negative coefficient turns the sign of an infinite one at every frame.)
template <bool REV>
__device__ __forceinline__ void onepole_carry_tags(int B, int T, int NT, float a, float *state, float *y,
                                                const unsigned long long *chain) {
  for (int b = 0; b < B; ++b) {
    const unsigned long long *cells = chain + 1 + (size_t)b * NT;
    float *yb = y + (size_t)b * T;
    int first = NT;
    for (int t = threadIdx.x; t < NT; t += OP_THREADS)
      if (dgchain::look(cells + t) & dgchain::TAG) {
        first = t;
        break;
      }
    __shared__ int lowest[OP_WARPS];
    first = __reduce_min_sync(0xffffffffu, first);
    if ((threadIdx.x & 31) == 0) lowest[threadIdx.x >> 5] = first;
    __syncthreads();
    for (int w = 0; w < OP_WARPS; ++w) first = min(first, lowest[w]);
    __syncthreads();
    if (first == NT) continue;
    const int64_t n1 = (int64_t)(first + 1) * OP_TILE;
    const float v = __ldcg(yb + (REV ? T - n1 : n1 - 1));
    for (int64_t n = n1 + threadIdx.x; n < T; n += OP_THREADS) {
      float *p = yb + (REV ? T - 1 - n : n);
      const float carried = a < 0.0f && ((n - n1) & 1) == 0 ? -v : v;
      if (fabsf(__ldcg(p)) <= 3.402823466e38f) {
        *p = carried;
        if (state && n == T - 1) state[b] = carried;
      }
    }
  }
}

// REV: the same scan run backwards in time, the adjoint recursion lam[n] = g[n] + a lam[n+1] of the filter's backward
// pass.  y may be x.  state (optional): per voice the state entering the first frame, and on return the one after the
// last.  The blocks stay: while a tile is scanned the loads of the block's next one are in flight and the ticket after
// that is being drawn, else every tile pays the ticket's, the loads' and the end values' latency one after the other.
template <bool REV>
__global__ void __launch_bounds__(OP_THREADS, OP_BLOCKS)
onepole_kernel(const float *x, int B, int T, int NT, const OnepolePowers pw, float *state, float *y,
               unsigned long long *__restrict__ chain, int32_t *status) {
  dgc_after_previous();
  __shared__ float warp_end[2][OP_WARPS];
  __shared__ float sh_in[2];
  __shared__ uint32_t sh_index[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t total = (uint32_t)B * (uint32_t)NT;
  constexpr float FINITE = 3.402823466e38f;
  if (tid == 0) {
    // the second ticket is drawn when the first has come: the blocks' first tiles are then all before their second ones
    const uint32_t first = dgchain::take_ticket(chain);
    sh_index[0] = first;
    sh_index[1] = first < total ? dgchain::take_ticket(chain) : total;
  }
  __syncthreads();
  uint32_t index = sh_index[0], next = sh_index[1];
  const float a = pw.a;
  float loc[OP_PER], ahead[OP_PER];
  if (index < total) {
    const int tile = (int)(index / (uint32_t)B), b = (int)(index - (uint32_t)tile * B);
    onepole_load<REV>(x + (size_t)b * T, T, tile * OP_TILE + tid * OP_PER, loc);
  }
  for (int par = 0; index < total; par ^= 1) {
    const int tile = (int)(index / (uint32_t)B), b = (int)(index - (uint32_t)tile * B);
    const int n0 = tile * OP_TILE + tid * OP_PER;
    unsigned long long *cells = chain + 1 + (size_t)b * NT;
    uint32_t after = total;
    if (next < total) {
      const int t1 = (int)(next / (uint32_t)B), b1 = (int)(next - (uint32_t)t1 * B);
      onepole_load<REV>(x + (size_t)b1 * T, T, t1 * OP_TILE + tid * OP_PER, ahead);
      if (tid == 0) after = dgchain::take_ticket(chain);
    }
    float prev = 0.0f;
#pragma unroll
    for (int j = 0; j < OP_PER; ++j) {
      prev = fmaf(a, prev, loc[j]);
      loc[j] = prev;
    }
    // state at the end of this thread's run, the tile started from rest: decayed scan over the warp, then over the warps
    float v = prev;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const float o = __shfl_up_sync(0xffffffffu, v, 1 << i);
      if (lane >= (1 << i)) v = fmaf(pw.r[i], o, v);
    }
    float excl = __shfl_up_sync(0xffffffffu, v, 1);
    if (lane == 0) excl = 0.0f;
    if (lane == 31) warp_end[par][warp] = v;
    __syncthreads();
    if (warp == 0) {
      float w = lane < OP_WARPS ? warp_end[par][lane] : 0.0f;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float o = __shfl_up_sync(0xffffffffu, w, 1 << i);
        if (lane >= (1 << i)) w = fmaf(pw.r[5 + i], o, w);
      }
      float in = 0.0f;
      if (tile == 0) {
        if (state) in = state[b];
        if (lane == OP_WARPS - 1 && NT > 1) dgchain::publish(cells, (float)(pw.tile[0] * (double)in + (double)w));
      } else {
        if (lane == OP_WARPS - 1 && tile < NT - 1) dgchain::publish(cells + tile, w);
        // sum over j of A^j end[tile - 1 - j]
        double decay = 1.0, acc = 0.0;
#pragma unroll
        for (int i = 0; i < 5; ++i)
          if (lane & (1 << i)) decay = fmin(decay * pw.tile[i], 1e300);
        const int far = min(tile, pw.reach);
        for (int j = lane; j < far; j += 32) {
          acc += decay * (double)dgchain::await(cells + tile - 1 - j, chain, status);
          decay = fmin(decay * pw.tile[5], 1e300);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        in = (float)acc;
        // the first tile has read the state cell before this, the last, tile writes it
        if (state && tile == NT - 1 && lane == 0) dgchain::await(cells, chain, status);
      }
      if (lane < OP_WARPS) warp_end[par][lane] = w;
      if (lane == 0) {
        sh_in[par] = in;
        sh_index[par] = after;
      }
    }
    __syncthreads();
    // state entering this thread's run: what its warp gathered, what the warps before left, what entered the tile
    float d = 1.0f;
#pragma unroll
    for (int i = 0; i < 5; ++i)
      if (lane & (1 << i)) d *= pw.r[i];
    if (warp > 0) excl = fmaf(d, warp_end[par][warp - 1], excl);
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (warp & (1 << i)) d *= pw.r[5 + i];
    float s = fmaf(d, sh_in[par], excl);
#pragma unroll
    for (int j = 0; j < OP_PER; ++j) {
      s *= a;
      loc[j] += s;
    }
    onepole_store<REV>(y + (size_t)b * T, T, n0, loc);
    if (state && tile == NT - 1) {
#pragma unroll
      for (int j = 0; j < OP_PER; ++j)
        if (n0 + j == T - 1) state[b] = loc[j];
    }
    if (tid == OP_THREADS - 1 && tile < NT - 1 && !(fabsf(loc[OP_PER - 1]) <= FINITE)) dgchain::tag(cells + tile, chain);
    index = next;
    next = sh_index[par];
#pragma unroll
    for (int j = 0; j < OP_PER; ++j) loc[j] = ahead[j];
  }
  __syncthreads();
  if (tid == 0) sh_index[0] = dgchain::last_with_tags(chain);
  __syncthreads();
  if (sh_index[0]) onepole_carry_tags<REV>(B, T, NT, a, state, y, chain);
}

// The filter in three launches: end value of every tile, the states entering the tiles, the output.  For filters that
// remember longer than OP_REACH tiles, and for a plan's step without a state cell (dgc_onepole_in_passes below).
template <bool REV, bool OUT>
__global__ void __launch_bounds__(OP_THREADS)
onepole_pass_kernel(const float *x, int T, int NT, const OnepolePowers pw, float *__restrict__ tiles, float *state, float *y) {
  dgc_after_previous();
  __shared__ float warp_end[OP_WARPS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b = blockIdx.x / NT, tile = blockIdx.x - b * NT;
  const size_t at = (size_t)b * T;
  const int n0 = tile * OP_TILE + tid * OP_PER;
  float loc[OP_PER], prev = 0.0f;
  onepole_load<REV>(x + at, T, n0, loc);
#pragma unroll
  for (int j = 0; j < OP_PER; ++j) loc[j] = prev = fmaf(pw.a, prev, loc[j]);
  float v = prev, d = 1.0f;
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const float o = __shfl_up_sync(0xffffffffu, v, 1 << i);
    if (lane >= (1 << i)) v = fmaf(pw.r[i], o, v);
    if (lane & (1 << i)) d *= pw.r[i];
  }
  if (lane == 31) warp_end[warp] = v;
  __syncthreads();
  float before = 0.0f;         // what the warps before left, the tile started from rest
  for (int w = 0; w < warp; ++w) before = fmaf(pw.r[5], before, warp_end[w]);
  if (!OUT) {
    if (tid == OP_THREADS - 1) tiles[blockIdx.x] = fmaf(pw.r[5], before, v);
    return;
  }
  float s = __shfl_up_sync(0xffffffffu, v, 1);
  s = fmaf(d, before, lane == 0 ? 0.0f : s);
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (warp & (1 << i)) d *= pw.r[5 + i];
  s = fmaf(d, tiles[blockIdx.x], s);
#pragma unroll
  for (int j = 0; j < OP_PER; ++j) {
    s *= pw.a;
    loc[j] += s;
  }
  onepole_store<REV>(y + at, T, n0, loc);
  if (state && tile == NT - 1) {
#pragma unroll
    for (int j = 0; j < OP_PER; ++j)
      if (n0 + j == T - 1) state[b] = loc[j];
  }
}

// The states entering the tiles, in double, a thread per voice with the next end values in flight
__global__ void __launch_bounds__(32)
onepole_carry_kernel(float *__restrict__ tiles, int B, int NT, double across, const float *__restrict__ state) {
  dgc_after_previous();
  constexpr int AHEAD = 32;
  const int b = blockIdx.x * 32 + threadIdx.x;
  if (b >= B) return;
  float *t = tiles + (size_t)b * NT;
  double s = state ? (double)state[b] : 0.0;
  float next[AHEAD];
  auto fetch = [&](int c0) {
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) next[j] = c0 + j < NT ? t[c0 + j] : 0.0f;
  };
  fetch(0);
  for (int c0 = 0; c0 < NT; c0 += AHEAD) {
    float end[AHEAD];
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) end[j] = next[j];
    fetch(c0 + AHEAD);
#pragma unroll
    for (int j = 0; j < AHEAD; ++j)
      if (c0 + j < NT) {
        t[c0 + j] = (float)s;
        s = across * s + (double)end[j];
      }
  }
}

template <bool REV>
void onepole_passes(cudaStream_t stream, const float *x, int B, int T, int NT, const OnepolePowers &pw, float *tiles, float *state,
                    float *y) {
  dgc_launch(onepole_pass_kernel<REV, false>, B * NT, OP_THREADS, 0, stream, x, T, NT, pw, tiles, nullptr, y);
  dgc_launch(onepole_carry_kernel, dgc_div_up(B, 32), 32, 0, stream, tiles, B, NT, pw.tile[0], state);
  dgc_launch(onepole_pass_kernel<REV, true>, B * NT, OP_THREADS, 0, stream, x, T, NT, pw, tiles, state, y);
}

template <bool REV>
int32_t launch_onepole_passes(dgc_ctx *ctx, const float *x, int B, int T, const OnepolePowers &pw, float *state, float *y,
                              const char *what) {
  const int NT = dgc_div_up(T, OP_TILE);
  float *tiles = dgc_ctx_scratch(ctx, (uint64_t)B * NT);
  if (!tiles) return DGC_ERR_OOM;
  onepole_passes<REV>(ctx->stream, x, B, T, NT, pw, tiles, state, y);
  ctx->launches += 3;
  return dgc_check_launch(ctx, what);
}

template <bool REV>
int32_t launch_onepole(dgc_ctx *ctx, const float *x, int B, int T, float a, float *state, float *y, const char *what) {
  const int NT = dgc_div_up(T, OP_TILE);
  const uint64_t tiles = (uint64_t)B * NT, room = (uint64_t)ctx->sm_count * OP_BLOCKS;
  DGC_REQUIRE(ctx, tiles <= 0x7fffffffull, "B * T too large");
  const OnepolePowers pw = onepole_powers(a);
  if (NT > OP_REACH && pw.reach > OP_REACH) return launch_onepole_passes<REV>(ctx, x, B, T, pw, state, y, what);
  unsigned long long *chain = dgc_ctx_chain(ctx, tiles);
  if (!chain) return DGC_ERR_OOM;
  dgc_launch(onepole_kernel<REV>, (unsigned)(tiles < room ? tiles : room), OP_THREADS, 0, ctx->stream, x, B, T, NT, pw, state, y,
             chain, ctx->status_dev);
  DGC_LAUNCHED(ctx, what);
  return DGC_OK;
}

// ---------------------------------------------------------------------------------------------
// biquad bank
// ---------------------------------------------------------------------------------------------
constexpr int BQ_CHUNK = 512;     // frames per (lane, chunk) thread
constexpr int BQ_THREADS = 128;   // lanes per block

// value with derivatives w.r.t. cutoff and q
struct Dual {
  float v, dc, dq;
};
__device__ __forceinline__ Dual dmul(Dual a, Dual b) { return {a.v * b.v, a.dc * b.v + a.v * b.dc, a.dq * b.v + a.v * b.dq}; }
__device__ __forceinline__ Dual dadd(Dual a, Dual b) { return {a.v + b.v, a.dc + b.dc, a.dq + b.dq}; }
__device__ __forceinline__ Dual dsub(Dual a, Dual b) { return {a.v - b.v, a.dc - b.dc, a.dq - b.dq}; }
__device__ __forceinline__ Dual ddiv(Dual a, Dual b) {
  float q = a.v / b.v;
  return {q, (a.dc - q * b.dc) / b.v, (a.dq - q * b.dq) / b.v};
}
__device__ __forceinline__ Dual dconst(float c) { return {c, 0.f, 0.f}; }
__device__ __forceinline__ Dual dabs(Dual a) { return a.v < 0.f ? Dual{-a.v, -a.dc, -a.dq} : a; }

__device__ __forceinline__ Dual dselect(float mode1, const Dual *opt, int n) {
  if (mode1 <= 0.f) return dconst(0.f);
  for (int i = 0; i < n; ++i)
    if (mode1 <= (float)(i + 1)) return opt[i];
  return dconst(0.f);
}

// Graph.biquad coefficient DAG (Sources/DGen/HigherOps.swift:444-555), all eight modes, node by node.
// coef layout per lane: b0 b1 b2 a1 a2, then d/dcutoff of the five, then d/dq of the five.
__device__ __noinline__ void biquad_coef(const float *__restrict__ cutoff, const float *__restrict__ q, int l, float gain,
                                         float mode, float *__restrict__ coef) {
  Dual cut = {cutoff[l], 1.f, 0.f}, res = {q[l], 0.f, 1.f};
  float add4 = mode + 1.0f;
  Dual mult7 = dmul(dabs(cut), dconst(0.00014247585730565955f));
  Dual cos8 = {cosf(mult7.v), -sinf(mult7.v) * mult7.dc, -sinf(mult7.v) * mult7.dq};
  Dual mult9 = dmul(cos8, dconst(-1.f));
  Dual add10 = dadd(mult9, dconst(1.f));
  Dual div11 = ddiv(add10, dconst(2.f));
  Dual sub12 = dsub(mult9, dconst(1.f));
  Dual div13 = ddiv(sub12, dconst(-2.f));
  Dual sin14 = {sinf(mult7.v), cosf(mult7.v) * mult7.dc, cosf(mult7.v) * mult7.dq};
  Dual mult15 = dmul(sin14, dconst(0.5f));
  Dual abs17 = dabs(res);
  Dual div18 = ddiv(mult15, abs17);
  Dual mult19 = dmul(div18, dconst(-1.f));
  Dual mult20 = dmul(div18, abs17);
  Dual mult21 = dmul(mult20, dconst(-1.f));
  Dual add22 = dadd(div18, dconst(1.f));
  Dual recip24 = ddiv(dconst(1.f), add22);
  Dual mult26 = dmul(recip24, dconst(gain));
  Dual mult31 = dmul(mult9, dconst(2.f));
  Dual not_sub35 = dsub(dconst(1.f), div18);
  // shelf coefficients, modes 6 (high shelf) and 7 (low shelf): HigherOps.swift:468-528; A depends on the gain only
  const float Af = sqrtf(fabsf(gain));
  Dual A = dconst(Af);
  Dual cosW0Pos = dmul(mult9, dconst(-1.f));
  Dual alphaShelf = ddiv(sin14, dmul(dconst(2.0f), abs17));
  Dual Ap1 = dconst(Af + 1.0f), Am1 = dconst(Af - 1.0f);
  Dual Ap1_cos = dmul(Ap1, cosW0Pos), Am1_cos = dmul(Am1, cosW0Pos);
  Dual tsa = dmul(dconst(2.0f * sqrtf(Af)), alphaShelf);
  Dual hs_b0 = dmul(A, dadd(dadd(Ap1, Am1_cos), tsa));
  Dual hs_b1 = dmul(dconst(-2.0f), dmul(A, dadd(Am1, Ap1_cos)));
  Dual hs_b2 = dmul(A, dsub(dadd(Ap1, Am1_cos), tsa));
  Dual hs_a0 = dadd(dsub(Ap1, Am1_cos), tsa);
  Dual ls_b0 = dmul(A, dadd(dsub(Ap1, Am1_cos), tsa));
  Dual ls_b1 = dmul(dconst(2.0f), dmul(A, dsub(Am1, Ap1_cos)));
  Dual ls_b2 = dmul(A, dsub(dsub(Ap1, Am1_cos), tsa));
  Dual ls_a0 = dadd(dadd(Ap1, Am1_cos), tsa);
  Dual hs_a1n = ddiv(dmul(dconst(2.0f), dsub(Am1, Ap1_cos)), hs_a0), hs_a2n = ddiv(dsub(dsub(Ap1, Am1_cos), tsa), hs_a0);
  Dual ls_a1n = ddiv(dmul(dconst(-2.0f), dadd(Am1, Ap1_cos)), ls_a0), ls_a2n = ddiv(dsub(dadd(Ap1, Am1_cos), tsa), ls_a0);
  Dual o23[8] = {div11, div13, mult19, mult21, dconst(1.f), add22, ddiv(hs_b2, hs_a0), ddiv(ls_b2, ls_a0)};
  Dual o32[8] = {add10, sub12, dconst(0.f), dconst(0.f), mult31, mult31, ddiv(hs_b1, hs_a0), ddiv(ls_b1, ls_a0)};
  Dual o36[8] = {div11, div13, div18, mult20, dconst(1.f), not_sub35, ddiv(hs_b0, hs_a0), ddiv(ls_b0, ls_a0)};
  // modes 0-5 scale by gain / a0; the shelves carry the gain in A (isShelfMode = mode >= 6, :533-548)
  const bool shelf = mode >= 6.0f;
  Dual s23 = dselect(add4, o23, 8), s32 = dselect(add4, o32, 8), s36 = dselect(add4, o36, 8);
  Dual b2 = shelf ? s23 : dmul(s23, mult26);
  Dual b1 = shelf ? s32 : dmul(s32, mult26);
  Dual b0 = shelf ? s36 : dmul(s36, mult26);
  Dual a2 = shelf ? (mode >= 7.0f ? ls_a2n : hs_a2n) : dmul(not_sub35, recip24);
  Dual a1 = shelf ? (mode >= 7.0f ? ls_a1n : hs_a1n) : dmul(mult31, recip24);
  float *c = coef + (size_t)l * 15;
  c[0] = b0.v; c[1] = b1.v; c[2] = b2.v; c[3] = a1.v; c[4] = a2.v;
  c[5] = b0.dc; c[6] = b1.dc; c[7] = b2.dc; c[8] = a1.dc; c[9] = a2.dc;
  c[10] = b0.dq; c[11] = b1.dq; c[12] = b2.dq; c[13] = a1.dq; c[14] = a2.dq;
}
__global__ void biquad_coef_kernel(const float *__restrict__ cutoff, const float *__restrict__ q, int L, float gain,
                                   float mode, float *__restrict__ coef) {
  dgc_after_previous();
  int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l < L) biquad_coef(cutoff, q, l, gain, mode, coef);
}

struct Coef {
  float b0, b1, b2, a1, a2;
};
__device__ __forceinline__ Coef load_coef(const float *coef, int l) {
  const float *c = coef + (size_t)l * 15;
  return {c[0], c[1], c[2], c[3], c[4]};
}

// y = ((b2*x2 + b1*x1) + b0*x0) - (a2*y2 + a1*y1), each operation rounded as in the reference graph
__device__ __forceinline__ float biquad_step(const Coef &c, float x0, float x1, float x2, float y1, float y2) {
  float add39 = __fadd_rn(__fadd_rn(__fmul_rn(x2, c.b2), __fmul_rn(x1, c.b1)), __fmul_rn(x0, c.b0));
  float add45 = __fadd_rn(__fmul_rn(y2, c.a2), __fmul_rn(y1, c.a1));
  return __fsub_rn(add39, add45);
}

// The samples x[c0 BQ_CHUNK - 2 ..] of the chunks that a block's consecutive (chunk, lane) pairs touch, staged in shared
// memory; returns this thread's pair, or false.  xc[n] is the chunk's frame n.  A bank of few lanes so fills its warps with
// several chunks (37 lanes left 91 of 128 threads without work).
__device__ __forceinline__ bool biquad_stage(const float *__restrict__ xb, int T, int L, int NC, float *sm, int &c, int &l,
                                             const float *&xc) {
  const int64_t i0 = (int64_t)blockIdx.x * blockDim.x, i = i0 + threadIdx.x, pairs = (int64_t)NC * L;
  const int c0 = (int)(i0 / L), c1 = (int)((min(i0 + blockDim.x, pairs) - 1) / L);
  const int span = (c1 - c0 + 1) * BQ_CHUNK + 2, t0 = c0 * BQ_CHUNK - 2;
  sm += 2;                                      // a chunk's frames start at a multiple of 16 bytes
  for (int j = threadIdx.x; j < span; j += blockDim.x) sm[j] = t0 + j >= 0 && t0 + j < T ? xb[t0 + j] : 0.0f;
  __syncthreads();
  if (i >= pairs) return false;
  c = (int)(i / L);
  l = (int)(i - (int64_t)c * L);
  xc = sm + (c - c0) * BQ_CHUNK + 2;
  return true;
}
// pairs per block (fewer where a bank of one lane would make a block's chunks too many for shared memory), staged bytes
int biquad_pairs(int L) { return L == 1 ? 64 : BQ_THREADS; }
int biquad_stage_bytes(int L) {
  const int n = biquad_pairs(L);
  return ((L % n == 0 ? 1 : n / L + 2) * BQ_CHUNK + 4) * (int)sizeof(float);
}

// Forward sweep.  PHASE 0: end state of every (voice, lane, chunk) from a zero y-state.
//                 PHASE 1: rerun from the carried state and write y[b][n][l] (lanes fastest).
template <int PHASE>
__global__ void __launch_bounds__(BQ_THREADS)
biquad_fwd_kernel(const float *__restrict__ x, const float *__restrict__ coef, int T, int L, int NC,
                  float *__restrict__ state /* [B][NC][L][2] */, float *__restrict__ y,
                  const float *__restrict__ st0 = nullptr /* [B][4][L]: history cells before the call */) {
  dgc_after_previous();
  extern __shared__ __align__(16) float sm[];
  const int b = blockIdx.y;
  int c, l;
  const float *xc;
  if (!biquad_stage(x + (size_t)b * T, T, L, NC, sm, c, l, xc)) return;
  const int n0 = c * BQ_CHUNK, len = min(BQ_CHUNK, T - n0);
  const Coef cf = load_coef(coef, l);
  float *st = state + (((size_t)b * NC + c) * L + l) * 2;
  float y1 = 0.f, y2 = 0.f;
  if (PHASE == 1) {
    y1 = st[0];
    y2 = st[1];
  }
  float x2 = xc[-2], x1 = xc[-1];
  if (st0 && c == 0) {   // x[-1], x[-2] come from the history cells
    x1 = st0[((size_t)b * 4 + 2) * L + l];
    x2 = st0[((size_t)b * 4 + 3) * L + l];
  }
  float *yo = y + ((size_t)b * T + n0) * L + l;
  auto step = [&](float x0) {
    const float v = biquad_step(cf, x0, x1, x2, y1, y2);
    if (PHASE == 1) {
      *yo = v;
      yo += L;
    }
    x2 = x1; x1 = x0; y2 = y1; y1 = v;
  };
  int n = 0;
  float4 next = *reinterpret_cast<const float4 *>(xc);   // four frames ahead of the recursion
#pragma unroll 2
  for (; n + 4 <= len; n += 4) {
    const float4 now = next;
    if (n + 8 <= len) next = *reinterpret_cast<const float4 *>(xc + n + 4);
    step(now.x);
    step(now.y);
    step(now.z);
    step(now.w);
  }
  for (; n < len; ++n) step(xc[n]);
  if (PHASE == 0) {
    st[0] = y1;
    st[1] = y2;
  }
}

// End state of a chunk as a LINEAR functional of its input.  Run from a zero y-state, the state (y[end], y[end-1])
// of lane l after a chunk is sum_m G[2l+s][m] * x[n0+m] plus two terms for the x-history x[n0-1], x[n0-2]:
//   hy[0] = 1, hy[k] = -a1 hy[k-1] - a2 hy[k-2]                  (response of the recursion to a unit drive)
//   h[k]  = b0 hy[k] + b1 hy[k-1] + b2 hy[k-2]                   (impulse response of the filter)
//   G[2l+0][m] = h[C-1-m], G[2l+1][m] = h[C-2-m]
//   history:  x[n0-1] -> (b1 hy[C-1] + b2 hy[C-2], b1 hy[C-2] + b2 hy[C-3]),  x[n0-2] -> (b2 hy[C-1], b2 hy[C-2])
// With that table the first pass of the forward -- the end state of EVERY (voice, chunk, lane) -- is one matrix
// product X[B*NC][C] * G^T[C][2L] on the tensor cores (its result lands directly in the [B][NC][L][2] state
// layout) instead of a second run of the serial recurrence.  The table is evaluated in double per call (the
// coefficients are inputs) and rounded once.
// Coefficients, the homogeneous transition M over one chunk, (y1, y2)_end = M (y1, y2)_start for zero input, and (G not null)
// the table, in one launch: a warp per lane, whose first two threads walk the recursion from (1, 0) -- those are the hy[k]
// -- and from (0, 1).  M's entries are large with cancelling signs where the poles are close to the unit circle: double.
// Bound by the walk, 512 dependent steps: 10.5 us for 256 lanes; 54 us when a thread per lane did all of it in three kernels
// and wrote its row of G value by value.
__global__ void __launch_bounds__(128)
biquad_tables_kernel(const float *__restrict__ cutoff, const float *__restrict__ q, int L, float gain, float mode,
                     float *__restrict__ coef, double *__restrict__ trans, float *__restrict__ G,
                     float *__restrict__ hist /* [L][4] */) {
  dgc_after_previous();
  __shared__ double hys[4][BQ_CHUNK + 2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l = blockIdx.x * 4 + warp;
  if (l >= L) return;
  if (lane == 0) biquad_coef(cutoff, q, l, gain, mode, coef);
  __syncwarp();
  const float *cp = coef + (size_t)l * 15;
  const double b0 = __ldcg(cp), b1 = __ldcg(cp + 1), b2 = __ldcg(cp + 2), a1 = __ldcg(cp + 3), a2 = __ldcg(cp + 4);
  double *hy = hys[warp] + 2;                  // hy[-2], hy[-1]: zero
  if (lane < 2) {
    const double n1 = -a1, n2 = -a2;           // the sign ahead of the products: one step less in the chain, the same value
    double y1 = lane == 0 ? 1.0 : 0.0, y2 = lane == 0 ? 0.0 : 1.0;
    if (lane == 0) {
      hy[-2] = hy[-1] = 0.0;
      hy[0] = 1.0;
    }
    for (int n = 0; n < BQ_CHUNK; n += 4) {    // the order of rounding of four steps as it always was, see BiquadSweep
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double v = j == 0 ? __fma_rn(n1, y1, __dmul_rn(n2, y2)) : __fma_rn(n2, y2, __dmul_rn(n1, y1));
        y2 = y1;
        y1 = v;
        if (lane == 0 && n + j + 1 < BQ_CHUNK) hy[n + j + 1] = v;
      }
    }
    trans[(size_t)l * 4 + lane] = y1;          // m11, m12
    trans[(size_t)l * 4 + 2 + lane] = y2;      // m21, m22
  }
  __syncwarp();
  if (!G) return;
  float *g1 = G + (size_t)(2 * l) * BQ_CHUNK, *g2 = g1 + BQ_CHUNK;
  for (int k = lane; k < BQ_CHUNK; k += 32) {
    const double h0 = hy[k], h1 = hy[k - 1], h2 = hy[k - 2];
    const float h = (float)(b0 * h0 + b1 * h1 + b2 * h2);
    // h[k] multiplies x[n0 + C-1-k] in y[end] and x[n0 + C-2-k] in y[end-1]
    g1[BQ_CHUNK - 1 - k] = h;
    if (k + 1 < BQ_CHUNK) g2[BQ_CHUNK - 2 - k] = h;
    else g2[BQ_CHUNK - 1] = 0.0f;              // m = C-1: h[-1] = 0
  }
  if (lane == 0) {
    const double y1 = hy[BQ_CHUNK - 1], y2 = hy[BQ_CHUNK - 2], y3 = hy[BQ_CHUNK - 3];
    hist[l * 4 + 0] = (float)(b1 * y1 + b2 * y2);
    hist[l * 4 + 1] = (float)(b1 * y2 + b2 * y3);
    hist[l * 4 + 2] = (float)(b2 * y1);
    hist[l * 4 + 3] = (float)(b2 * y2);
  }
}

// The same sweep with FOUR lanes per thread (L a multiple of 4): four independent recurrences hide the
// latency of the dependent multiply-adds of one, and the output goes out as one 128-bit store per frame and
// thread (a warp writes 512 contiguous bytes).  Block = (L/4 lane quads, up to 4 chunks).
constexpr int BQ4_CHUNKS = 4;
template <int PHASE>
__global__ void __launch_bounds__(256)
biquad_fwd4_kernel(const float *__restrict__ x, const float *__restrict__ coef, int B, int T, int L, int NC,
                   float *__restrict__ state /* [B][NC][L][2] */, float *__restrict__ y,
                   const float *__restrict__ st0 = nullptr /* [B][4][L]: history cells before the call */) {
  dgc_after_previous();
  __shared__ float xs[BQ4_CHUNKS][BQ_CHUNK + 2];
  const int lq = blockIdx.x * blockDim.x + threadIdx.x, cy = threadIdx.y;
  const int c = blockIdx.y * BQ4_CHUNKS + cy, b = blockIdx.z;
  const bool chunk_ok = c < NC;
  const float *xb = x + (size_t)b * T;
  const int n0 = c * BQ_CHUNK, len = chunk_ok ? min(BQ_CHUNK, T - n0) : 0;
  for (int i = threadIdx.x; i < len + 2; i += blockDim.x) {
    int t = n0 - 2 + i;
    xs[cy][i] = t >= 0 ? xb[t] : 0.0f;
  }
  __syncthreads();
  if (!chunk_ok || 4 * lq >= L) return;
  Coef cf[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) cf[k] = load_coef(coef, 4 * lq + k);
  float *st = state + (((size_t)b * NC + c) * L + 4 * lq) * 2;
  float y1[4] = {0.f, 0.f, 0.f, 0.f}, y2[4] = {0.f, 0.f, 0.f, 0.f};
  if (PHASE == 1) {
    const float4 s0 = *reinterpret_cast<const float4 *>(st), s1 = *reinterpret_cast<const float4 *>(st + 4);
    y1[0] = s0.x; y2[0] = s0.y; y1[1] = s0.z; y2[1] = s0.w;
    y1[2] = s1.x; y2[2] = s1.y; y1[3] = s1.z; y2[3] = s1.w;
  }
  float x2 = xs[cy][0], x1 = xs[cy][1];
  if (st0 && c == 0) {   // x[-1], x[-2] come from the history cells (one input feeds all lanes: the first lane's)
    x1 = st0[((size_t)b * 4 + 2) * L + 4 * lq];
    x2 = st0[((size_t)b * 4 + 3) * L + 4 * lq];
  }
  float *yo = y + ((size_t)b * T + n0) * L + 4 * lq;
#pragma unroll 2
  for (int n = 0; n < len; ++n) {
    const float x0 = xs[cy][n + 2];
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = biquad_step(cf[k], x0, x1, x2, y1[k], y2[k]);
      y2[k] = y1[k];
      y1[k] = v[k];
    }
    if (PHASE == 1) __stcs(reinterpret_cast<float4 *>(yo + (size_t)n * L), make_float4(v[0], v[1], v[2], v[3]));
    x2 = x1;
    x1 = x0;
  }
  if (PHASE == 0) {
    *reinterpret_cast<float4 *>(st) = make_float4(y1[0], y2[0], y1[1], y2[1]);
    *reinterpret_cast<float4 *>(st + 4) = make_float4(y1[2], y2[2], y1[3], y2[3]);
  }
}

// state[c] <- state entering chunk c: the affine maps s <- M s + e one after the other, in double, a thread per (voice, lane).
// The next BQ_AHEAD chunks are in flight while the present ones are walked.  Not a scan by runs: a last-bit change of a
// state is 140 times as much in the output of a low, sharp lane, and 10000 times in the gradient of its cutoff.
// hist (optional): the end states come from the matrix product, which knows nothing of the x-history before a chunk: its
// two terms are added here.  Bound by the instructions of a lone warp: pointers that step and no tests in a whole run of chunks,
// 32 voices x 512 chunks x 256 lanes 70 -> 25 us, 5 x 98 x 37 14 -> 6.
constexpr int BQ_AHEAD = 16;
__global__ void __launch_bounds__(32)
biquad_carry_kernel(const double *__restrict__ trans, const float *__restrict__ x, const float *__restrict__ hist, int T, int L,
                    int NC, float2 *__restrict__ state, const float *__restrict__ st0) {
  dgc_after_previous();
  const int l = blockIdx.x * 32 + threadIdx.x, b = blockIdx.y;
  if (l >= L) return;
  const double m11 = trans[(size_t)l * 4], m12 = trans[(size_t)l * 4 + 1], m21 = trans[(size_t)l * 4 + 2],
               m22 = trans[(size_t)l * 4 + 3];
  float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
  if (hist) h = make_float4(hist[l * 4], hist[l * 4 + 1], hist[l * 4 + 2], hist[l * 4 + 3]);
  const float *xb = x + (size_t)b * T;
  float2 *st = state + (size_t)b * NC * L + l;
  // y[-1], y[-2]: the history cells before the call, else rest
  double s1 = st0 ? (double)st0[((size_t)b * 4 + 0) * L + l] : 0.0, s2 = st0 ? (double)st0[((size_t)b * 4 + 1) * L + l] : 0.0;
  float2 e[BQ_AHEAD], xx[BQ_AHEAD];
  const float2 *pe = st;                     // where the next chunks' end states lie, the last frames before them, their states
  const float *px = xb - 2;
  float2 *ps = st;
  auto fetch = [&](int c0, auto whole) {
#pragma unroll
    for (int j = 0; j < BQ_AHEAD; ++j, pe += L, px += BQ_CHUNK) {
      if (decltype(whole)::value || c0 + j < NC) {
        e[j] = *pe;
        if (hist && c0 + j > 0) xx[j] = make_float2(__ldg(px + 1), __ldg(px));
      }
    }
    if (hist && c0 == 0 && st0) xx[0] = make_float2(st0[((size_t)b * 4 + 2) * L + l], st0[((size_t)b * 4 + 3) * L + l]);
  };
  auto walk = [&](int c0, auto whole) {
    float2 v[BQ_AHEAD];
#pragma unroll
    for (int j = 0; j < BQ_AHEAD; ++j) {
      v[j] = e[j];
      if (hist && (c0 + j > 0 || st0)) {
        v[j].x += h.x * xx[j].x + h.z * xx[j].y;
        v[j].y += h.y * xx[j].x + h.w * xx[j].y;
      }
    }
    if (c0 + 2 * BQ_AHEAD <= NC) fetch(c0 + BQ_AHEAD, std::true_type());
    else fetch(c0 + BQ_AHEAD, std::false_type());
#pragma unroll
    for (int j = 0; j < BQ_AHEAD; ++j, ps += L) {
      if (decltype(whole)::value || c0 + j < NC) {
        *ps = make_float2((float)s1, (float)s2);
        // every chunk but possibly the last has full length; the state after the last chunk is unused
        const double e1 = v[j].x, e2 = v[j].y;
        const double n1 = m11 * s1 + m12 * s2 + e1, n2 = m21 * s1 + m22 * s2 + e2;
        s1 = n1;
        s2 = n2;
      }
    }
  };
  fetch(0, std::false_type());
  int c0 = 0;
  for (; c0 + BQ_AHEAD <= NC; c0 += BQ_AHEAD) walk(c0, std::true_type());
  if (c0 < NC) walk(c0, std::false_type());
}

// Backward sweep for loss = scale * sum (y - t)^2.  Adjoint recurrence (transposed filter, reverse time):
//   lam[n] = g[n] - a1*lam[n+1] - a2*lam[n+2],  g = 2*scale*(y - t)
//   dL/db0 = sum lam[n] x[n], dL/db1 = sum lam[n] x[n-1], dL/db2 = sum lam[n] x[n-2],
//   dL/da1 = -sum lam[n] y[n-1], dL/da2 = -sum lam[n] y[n-2].
// One sweep per (voice, lane, chunk) from a zero terminal adjoint accumulates the five sums for the
// local adjoint AND for the two homogeneous adjoint responses h1, h2 (terminal state (1,0) and (0,1));
// the carry kernel then supplies the true terminal state s of each chunk and the total is
// S_loc + s1*S_h1 + s2*S_h2.  Record per (voice, chunk, lane): 15 sums + local start adjoint (2) + sq error.
constexpr int BW_REC = 18;

// The order in which a1 p + a2 q is rounded is spelled out: lam and one frame in sixteen (in the edge chunks every odd one)
// multiply a2 q first, the rest a1 p.  The gradient of a low cutoff is a difference of these sums that loses four digits,
// so another order is another gradient there (6e-3 at 32 voices x 256 lanes); this one is kept as it is.
__device__ __forceinline__ float feedback(const Coef &c, float p, float q, bool a2_first) {
  return a2_first ? __fmaf_rn(c.a1, p, __fmul_rn(c.a2, q)) : __fmaf_rn(c.a2, q, __fmul_rn(c.a1, p));
}

// a response of the adjoint recurrence to a terminal state (lam[n_end+1], lam[n_end+2]) = (p, q), and its five sums
struct BiquadResponse {
  float p, q;
  float S[5] = {};
  __device__ __forceinline__ BiquadResponse(float p, float q) : p(p), q(q) {}
  __device__ __forceinline__ void step(const Coef &cf, float x0, float x1, float x2, float ym1, float ym2, bool a2_first) {
    const float h = -feedback(cf, p, q, a2_first);
    S[0] = fmaf(h, x0, S[0]); S[1] = fmaf(h, x1, S[1]); S[2] = fmaf(h, x2, S[2]);
    S[3] = fmaf(h, ym1, S[3]); S[4] = fmaf(h, ym2, S[4]);
    q = p; p = h;
  }
  __device__ __forceinline__ void record(float *r, int L) const {
#pragma unroll
    for (int i = 0; i < 5; ++i) r[(size_t)i * L] = S[i];
  }
};

// the local adjoint from rest, its sums, the squared error
template <bool UP>
struct BiquadAdjoint {
  float la1 = 0.f, la2 = 0.f;                // lam[n+1], lam[n+2]
  float S[5] = {}, sq = 0.f;
  __device__ __forceinline__ void step(const Coef &cf, float gscale, float x0, float x1, float x2, float yc, float ym1, float ym2,
                                       float tv) {
    const float fed = feedback(cf, la1, la2, true), d = UP ? 0.0f : __fsub_rn(yc, tv);
    if (!UP) sq = fmaf(d, d, sq);
    const float lam = UP ? __fsub_rn(tv, fed) : __fmaf_rn(gscale, d, -fed);
    S[0] = fmaf(lam, x0, S[0]); S[1] = fmaf(lam, x1, S[1]); S[2] = fmaf(lam, x2, S[2]);
    S[3] = fmaf(lam, ym1, S[3]); S[4] = fmaf(lam, ym2, S[4]);
    la2 = la1; la1 = lam;
  }
  __device__ __forceinline__ void record(float *r, int L) const {
#pragma unroll
    for (int i = 0; i < 5; ++i) r[(size_t)i * L] = S[i];
    r[(size_t)15 * L] = la1;  // local adjoint at the first frame of the chunk: lam[n0]
    r[(size_t)16 * L] = la2;  // lam[n0+1]
    r[(size_t)17 * L] = sq;
  }
};

template <bool UP>
struct BiquadSweep {
  Coef cf;
  float gscale, yc, ym1;                     // y[n], y[n-1]
  BiquadAdjoint<UP> adj;
  BiquadResponse h1{1.f, 0.f}, h2{0.f, 1.f};

  // frame n: x[n], x[n-1], x[n-2], y[n-2], target
  __device__ __forceinline__ void step(float x0, float x1, float x2, float ym2, float tv, bool a2_first) {
    adj.step(cf, gscale, x0, x1, x2, yc, ym1, ym2, tv);
    h1.step(cf, x0, x1, x2, ym1, ym2, a2_first);
    h2.step(cf, x0, x1, x2, ym1, ym2, a2_first);
    yc = ym1; ym1 = ym2;
  }
  __device__ __forceinline__ void record(float *r, int L) const {
    adj.record(r, L);
    h1.record(r + (size_t)5 * L, L);
    h2.record(r + (size_t)10 * L, L);
  }
};

// UP = false: g = gscale * (y - tgt) (the MSE loss, squared error summed on the way);  UP = true: `tgt` IS the
// upstream gradient dL/dy [B][T][L] of an arbitrary loss.
// A group of sixteen frames issues its 32 loads before the dependent recurrence steps: the sweep is bound by loads in
// flight (32 voices x 262144 x 256 lanes: 17.2 GB in 3.12 ms, 84 % of the copy rate; 3.58 with 116 registers, a block less on an
// SM, when the frames of x were read one by one).  In the first and the last chunk frames
// outside the chunk or the signal are zeros.  A small bank takes as long as its slowest warp: only the groups that reach out of
// the chunk test their frames, and a warp with lanes of an edge chunk and of others walks them together; testing every frame,
// one kind after the other, 5 voices x 50001 x 37 lanes took 75 us, now 35.  A thread each for the adjoint and the two
// responses there: 3 us less at 145 blocks, 20 % more at 384.  Asynchronous copies to a ring in
// shared memory were measured: 6 % slower on the large bank.
template <bool UP>
__global__ void __launch_bounds__(BQ_THREADS)
biquad_bwd_kernel(const float *__restrict__ x, const float *__restrict__ coef, const float *__restrict__ y,
                  const float *__restrict__ tgt, int T, int L, int NC, float gscale,
                  float *__restrict__ rec /* [B][NC][BW_REC][L] */) {
  dgc_after_previous();
  extern __shared__ __align__(16) float sm[];   // staged frames are read four at a time
  constexpr int G = 16;
  const int b = blockIdx.y;
  int c, l;
  const float *xc;
  if (!biquad_stage(x + (size_t)b * T, T, L, NC, sm, c, l, xc)) return;
  const int n0 = c * BQ_CHUNK, len = min(BQ_CHUNK, T - n0);
  const float *yb = y + ((size_t)b * T + n0) * L + l, *tb = tgt + ((size_t)b * T + n0) * L + l;
  auto y_at = [&](int n) { return n0 + n >= 0 ? yb[(ptrdiff_t)n * L] : 0.0f; };
  BiquadSweep<UP> w{load_coef(coef, l), gscale, y_at(len - 1), y_at(len - 2)};
  // edge chunks: the first, whose frames reach back before the signal, and a short last one
  const bool edge = len < BQ_CHUNK || n0 < 2;
  auto group = [&](int nb, auto whole, auto any_edge) {   // whole: no frame of it outside the chunk or before the signal
    float yv[G], tv[G];
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const int n = nb + j;
      yv[j] = decltype(whole)::value || (n < len && n0 + n >= 2) ? __ldcs(yb + (ptrdiff_t)(n - 2) * L) : 0.0f;
      tv[j] = decltype(whole)::value || n < len ? __ldcs(tb + (ptrdiff_t)n * L) : 0.0f;
    }
    float xv[G + 2];                            // x[nb - 2 .. nb + G)
    {
      const float2 q = *reinterpret_cast<const float2 *>(xc + nb - 2);
      xv[0] = q.x; xv[1] = q.y;
    }
#pragma unroll
    for (int j = 0; j < G; j += 4) {
      const float4 q = *reinterpret_cast<const float4 *>(xc + nb + j);
      xv[j + 2] = q.x; xv[j + 3] = q.y; xv[j + 4] = q.z; xv[j + 5] = q.w;
    }
    const bool last = nb == BQ_CHUNK - G;
#pragma unroll
    for (int j = G - 1; j >= 0; --j) {
      const bool a2_first = j == G - 1 || (decltype(any_edge)::value && edge ? (j & 1) != 0 : j == G - 2 && last);
      if (decltype(whole)::value || nb + j < len) w.step(xv[j + 2], xv[j + 1], xv[j], yv[j], tv[j], a2_first);
    }
  };
  if (__any_sync(__activemask(), edge)) {
    for (int nb = BQ_CHUNK - G; nb >= 0; nb -= G) {
      if (nb + G <= len && n0 + nb >= 2) group(nb, std::true_type(), std::true_type());
      else if (nb < len) group(nb, std::false_type(), std::true_type());
    }
  } else {
    group(BQ_CHUNK - G, std::true_type(), std::false_type());
    for (int nb = BQ_CHUNK - 2 * G; nb >= 0; nb -= G) group(nb, std::true_type(), std::false_type());
  }
  w.record(rec + ((size_t)b * NC + c) * BW_REC * L + l, L);
}

struct Mat2 {
  double a, b, c, d;      // [[a, b], [c, d]]
};
__device__ __forceinline__ Mat2 mat_mul(const Mat2 &p, const Mat2 &q) {
  return {p.a * q.a + p.b * q.c, p.a * q.b + p.b * q.d, p.c * q.a + p.d * q.c, p.c * q.b + p.d * q.d};
}
// m^n by squaring
__device__ __forceinline__ Mat2 mat_pow(Mat2 m, int n) {
  Mat2 r = {1.0, 0.0, 0.0, 1.0};
  for (; n > 0; n >>= 1) {
    if (n & 1) r = mat_mul(r, m);
    m = mat_mul(m, m);
  }
  return r;
}

// Reverse carry over chunks, in double: resolves the terminal adjoint of every chunk, combines the sums, and writes per
// (voice, lane) the five coefficient-gradient sums and the squared error.  Block = 32 lanes of a voice x BQ_RUNS warps: a
// warp walks its run of consecutive chunks from rest, the ends of the runs are carried over by A^run, and the warp walks
// its run again from the true terminal adjoint; the warps' sums are added in a fixed order.  (Nothing here is rounded to
// single precision but the results.)  32 voices x 512 chunks x 256 lanes: 80 us, the record's 302 MB at 3.8 TB/s; 914 us when
// a thread per (voice, lane) walked all chunks, two warps on an SM.
constexpr int BQ_RUNS = 16;
__global__ void __launch_bounds__(32 * BQ_RUNS)
biquad_bwd_carry_kernel(const float *__restrict__ rec, const float *__restrict__ coef, int L, int NC,
                        double *__restrict__ acc /* [B][L][6] */, float2 *__restrict__ term /* [B][NC][L] or null */) {
  dgc_after_previous();
  __shared__ double2 ends[BQ_RUNS][32];
  __shared__ double sums[BQ_RUNS][6][32];
  const int l = blockIdx.x * 32 + threadIdx.x, run = threadIdx.y, b = blockIdx.y;
  // run 0 takes the LAST chunks, the ones the reverse pass meets first
  const int per = (NC + BQ_RUNS - 1) / BQ_RUNS, d0 = min(run * per, NC), d1 = min(d0 + per, NC);
  const bool live = l < L;
  const Coef cf = live ? load_coef(coef, l) : Coef{};
  const float *rb = rec + (size_t)b * NC * BW_REC * L + l;
  // (lam[n0], lam[n0+1]) = A (terminal adjoint) + local, A = [[h1[0], h2[0]], [h1[1], h2[1]]] over a full chunk.  The one
  // chunk that may be shorter is the last, whose terminal adjoint is zero.
  const Mat2 A = mat_pow({-(double)cf.a1, -(double)cf.a2, 1.0, 0.0}, BQ_CHUNK);
  double s1 = 0.0, s2 = 0.0;
  if (live) {
#pragma unroll 8
    for (int d = d0; d < d1; ++d) {
      const float *r = rb + (size_t)(NC - 1 - d) * BW_REC * L;
      const double n1 = A.a * s1 + A.b * s2 + (double)r[(size_t)15 * L], n2 = A.c * s1 + A.d * s2 + (double)r[(size_t)16 * L];
      s1 = n1;
      s2 = n2;
    }
  }
  ends[run][threadIdx.x] = make_double2(s1, s2);
  __syncthreads();
  double g[6] = {0, 0, 0, 0, 0, 0};
  if (live && d0 < d1) {
    s1 = s2 = 0.0;
    const Mat2 Ar = mat_pow(A, per);
    for (int q = 0; q < run; ++q) {
      const double2 e = ends[q][threadIdx.x];
      const double n1 = Ar.a * s1 + Ar.b * s2 + e.x, n2 = Ar.c * s1 + Ar.d * s2 + e.y;
      s1 = n1;
      s2 = n2;
    }
#pragma unroll 2
    for (int d = d0; d < d1; ++d) {
      const int c = NC - 1 - d;
      const float *r = rb + (size_t)c * BW_REC * L;
      if (term) term[((size_t)b * NC + c) * L + l] = make_float2((float)s1, (float)s2);
#pragma unroll
      for (int i = 0; i < 5; ++i)
        g[i] += (double)r[(size_t)i * L] + s1 * (double)r[(size_t)(5 + i) * L] + s2 * (double)r[(size_t)(10 + i) * L];
      g[5] += (double)r[(size_t)17 * L];
      const double n1 = A.a * s1 + A.b * s2 + (double)r[(size_t)15 * L], n2 = A.c * s1 + A.d * s2 + (double)r[(size_t)16 * L];
      s1 = n1;
      s2 = n2;
    }
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) sums[run][i][threadIdx.x] = g[i];
  __syncthreads();
  if (live && run < 6) {
    double t = 0.0;
    for (int q = 0; q < BQ_RUNS; ++q) t += sums[q][run][threadIdx.x];
    acc[((size_t)b * L + l) * 6 + run] = run == 3 || run == 4 ? -t : t;
  }
}

// Gradient with respect to the INPUT x[b][n] (shared by the lanes): sum over lanes of
//   b0 lam[n] + b1 lam[n+1] + b2 lam[n+2]
// A second reverse sweep per (voice, lane, chunk), now from the chunk's TRUE terminal adjoint (resolved by the carry
// kernel), recomputes lam; the sum over the block's 128 lanes goes through a shared-memory tile of 32 frames, the
// sum over lane blocks through per-block partial rows that a last kernel adds in a fixed order.
// Bound by the walk's instructions: no tests in a whole group of frames, a pointer that steps, nothing to walk for a warp
// without lanes, a quarter of the lanes per warp in the sums: 5 voices x 50001 x 37 lanes 42 -> 24.5 us, 300 lanes 120 -> 80.
// (The next group's loads sent ahead in registers: 46 and 115; by asynchronous copies: 22 us there, 7 % slower with 100 lanes.)
constexpr int GX_FRAMES = 32;

__global__ void __launch_bounds__(BQ_THREADS)
biquad_gx_kernel(const float *__restrict__ coef, const float *__restrict__ gy, const float2 *__restrict__ term, int B, int T,
                 int L, int NC,
                 float *__restrict__ part /* [gridDim.x][B][T] */) {
  dgc_after_previous();
  __shared__ float red[GX_FRAMES][BQ_THREADS + 1];
  __shared__ float quarter[4][GX_FRAMES];
  const int quarters = min(4, (L - (int)blockIdx.x * BQ_THREADS + 31) / 32);   // those with lanes
  const int tid = threadIdx.x, l = blockIdx.x * BQ_THREADS + tid, c = blockIdx.y, b = blockIdx.z;
  const int n0 = c * BQ_CHUNK, len = min(BQ_CHUNK, T - n0);
  const bool live = l < L;
  Coef cf = {};
  float la1 = 0.f, la2 = 0.f;
  if (live) {
    cf = load_coef(coef, l);
    const float2 s = term[((size_t)b * NC + c) * L + l];
    la1 = s.x;
    la2 = s.y;
  }
  const float *gb = gy + ((size_t)b * T + n0) * L + l;
  float *pb = part + ((size_t)blockIdx.x * B + b) * T;
  if (!live)
    for (int j = 0; j < GX_FRAMES; ++j) red[j][tid] = 0.f;
  // groups of 32 frames from the end of the chunk; the last group (lowest frames) may be shorter
  for (int hi = len; hi > 0; hi -= GX_FRAMES) {
    const int lo = max(hi - GX_FRAMES, 0), cnt = hi - lo;
    auto walk = [&](auto whole) {
      float gv[GX_FRAMES];
      const float *p = gb + (size_t)lo * L;
#pragma unroll
      for (int j = 0; j < GX_FRAMES; ++j, p += L) gv[j] = decltype(whole)::value || j < cnt ? __ldcs(p) : 0.f;
#pragma unroll
      for (int j = GX_FRAMES - 1; j >= 0; --j) {
        float contrib = 0.f;
        if (decltype(whole)::value || j < cnt) {
          const float lam = __fsub_rn(gv[j], fmaf(cf.a1, la1, __fmul_rn(cf.a2, la2)));
          contrib = fmaf(cf.b0, lam, fmaf(cf.b1, la1, cf.b2 * la2));
          la2 = la1;
          la1 = lam;
        }
        red[j][tid] = contrib;
      }
    };
    if (live) {
      if (cnt == GX_FRAMES) walk(std::true_type());
      else walk(std::false_type());
    }
    __syncthreads();
    // warp -> quarter of the lanes, thread -> frame: 32 adds, then the four quarters
    {
      const int j = tid & 31, seg = tid >> 5;
      float sum = 0.f;
      if (seg < quarters) {
#pragma unroll 8
        for (int k = 0; k < BQ_THREADS / 4; ++k)
          sum += red[j][seg * (BQ_THREADS / 4) + ((k + 4 * j + seg) & (BQ_THREADS / 4 - 1))];
      }
      quarter[seg][j] = sum;
    }
    __syncthreads();
    if (tid < cnt) pb[n0 + lo + tid] = (quarter[0][tid] + quarter[1][tid]) + (quarter[2][tid] + quarter[3][tid]);
  }
}

__global__ void sum_partial_rows_kernel(const float *__restrict__ part, int nparts, size_t n, float *__restrict__ out) {
  dgc_after_previous();
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = 0.f;
  for (int p = 0; p < nparts; ++p) s += part[(size_t)p * n + i];
  out[i] = s;
}

// Sum over voices, chain rule to cutoff and q, total loss: a warp per lane, the voices over its threads and a fixed tree;
// the block that finishes last adds the lanes' losses.
__global__ void __launch_bounds__(256)
biquad_bwd_final_kernel(const double *__restrict__ acc, const float *__restrict__ coef, int B, int L,
                        float loss_scale, float *__restrict__ gcut, float *__restrict__ gq,
                        double *__restrict__ lane_loss, unsigned int *__restrict__ ticket, double *__restrict__ loss) {
  dgc_after_previous();
  const int l = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (l < L) {
    double G[6] = {0, 0, 0, 0, 0, 0};
    for (int b = lane; b < B; b += 32)
#pragma unroll
      for (int i = 0; i < 6; ++i) G[i] += acc[((size_t)b * L + l) * 6 + i];
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) G[i] += __shfl_xor_sync(0xffffffffu, G[i], o);
    if (lane == 0) {
      const float *c = coef + (size_t)l * 15;
      double dc = 0, dq = 0;
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        dc += G[i] * (double)c[5 + i];
        dq += G[i] * (double)c[10 + i];
      }
      gcut[l] = (float)dc;
      gq[l] = (float)dq;
      lane_loss[l] = G[5] * (double)loss_scale;
    }
  }
  if (!loss) return;
  __shared__ bool last;
  __shared__ double part[256];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  double t = 0.0;
  for (int i = threadIdx.x; i < L; i += 256) t += __ldcg(lane_loss + i);
  part[threadIdx.x] = t;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *loss = part[0];
    *ticket = 0u;
  }
}

}  // namespace

DGC_EXPORT int32_t dgc_onepole_fwd(dgc_ctx *ctx, const float *x_dev, int32_t B, int32_t T, float a, float *y_dev) {
  return dgc_onepole_fwd_state(ctx, x_dev, B, T, a, nullptr, y_dev);
}

DGC_EXPORT int32_t dgc_onepole_fwd_state(dgc_ctx *ctx, const float *x_dev, int32_t B, int32_t T, float a,
                                         float *state_dev, float *y_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, x_dev && y_dev, "null pointer");
  DGC_REQUIRE(ctx, B > 0 && T > 0, "size out of range");
  return launch_onepole<false>(ctx, x_dev, B, T, a, state_dev, y_dev, "onepole");
}

int32_t dgc_onepole_in_passes(dgc_ctx *ctx, const float *x_dev, int32_t B, int32_t T, float a, float *y_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, x_dev && y_dev, "null pointer");
  DGC_REQUIRE(ctx, B > 0 && T > 0, "size out of range");
  DGC_REQUIRE(ctx, (uint64_t)B * dgc_div_up(T, OP_TILE) <= 0x7fffffffull, "B * T too large");
  return launch_onepole_passes<false>(ctx, x_dev, B, T, onepole_powers(a), nullptr, y_dev, "onepole");
}

static int32_t biquad_validate(dgc_ctx *ctx, const dgc_biquad_params *p) {
  DGC_REQUIRE(ctx, p->B > 0 && p->T > 0 && p->L > 0, "size out of range");
  DGC_REQUIRE(ctx, p->B <= 65535, "B must be <= 65535");
  DGC_REQUIRE(ctx, p->mode >= 0.0f && p->mode <= 7.0f, "mode must be in 0..7");
  return DGC_OK;
}

DGC_EXPORT uint64_t dgc_biquad_scratch_floats(const dgc_biquad_params *p, int32_t backward) {
  if (!p || p->B <= 0 || p->T <= 0 || p->L <= 0) return 0;
  uint64_t NC = (uint64_t)(p->T + BQ_CHUNK - 1) / BQ_CHUNK;
  uint64_t coef = (((uint64_t)p->L * 16 + (uint64_t)p->L * 8) + 3) & ~3ull;
  // forward: chunk states, then the end-state response table [2L][BQ_CHUNK] and its 4L history terms
  if (!backward) return coef + (((uint64_t)p->B * NC * p->L * 2 + 3) & ~3ull) + (uint64_t)p->L * (2 * BQ_CHUNK + 4) + 16;
  uint64_t rec = (uint64_t)p->B * NC * BW_REC * p->L;
  uint64_t base = coef + ((rec + 3) & ~3ull) + 2 * ((uint64_t)p->B * p->L * 6 + p->L) + 16;
  if (backward == 1) return base;
  // backward == 2 (dgc_biquad_bwd with the input gradient): terminal adjoints [B][NC][L] float2, partial rows
  uint64_t blocks = ((uint64_t)p->L + BQ_THREADS - 1) / BQ_THREADS;
  return base + 2 * (uint64_t)p->B * NC * p->L + blocks * (uint64_t)p->B * p->T + 16;
}

// history cells after the call: y[T-1], y[T-2], x[T-1], x[T-2] per (voice, lane); frames before the call come
// from the cells as they were
__global__ void biquad_final_state_kernel(const float *__restrict__ x, const float *__restrict__ y, int B, int T, int L,
                                          float *__restrict__ st) {
  dgc_after_previous();
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= B * L) return;
  const int b = idx / L, l = idx - b * L;
  float *s = st + (size_t)b * 4 * L + l;
  const float *yb = y + (size_t)b * T * L + l, *xb = x + (size_t)b * T;
  const float oy1 = s[0], ox1 = s[2 * L];
  s[0] = yb[(size_t)(T - 1) * L];
  s[L] = T >= 2 ? yb[(size_t)(T - 2) * L] : oy1;
  s[2 * L] = xb[T - 1];
  s[3 * L] = T >= 2 ? xb[T - 2] : ox1;
}

static int32_t biquad_fwd_impl(dgc_ctx *ctx, const dgc_biquad_params *p, const float *x_dev, const float *cutoff_dev,
                               const float *q_dev, float *scratch_dev, float *st0, float *y_dev);

DGC_EXPORT int32_t dgc_biquad_fwd(dgc_ctx *ctx, const dgc_biquad_params *p, const float *x_dev,
                                  const float *cutoff_dev, const float *q_dev, float *scratch_dev, float *y_dev) {
  return biquad_fwd_impl(ctx, p, x_dev, cutoff_dev, q_dev, scratch_dev, nullptr, y_dev);
}

DGC_EXPORT int32_t dgc_biquad_fwd_state(dgc_ctx *ctx, const dgc_biquad_params *p, const float *x_dev,
                                        const float *cutoff_dev, const float *q_dev, float *scratch_dev,
                                        float *state_dev, float *y_dev) {
  return biquad_fwd_impl(ctx, p, x_dev, cutoff_dev, q_dev, scratch_dev, state_dev, y_dev);
}

static int32_t biquad_fwd_impl(dgc_ctx *ctx, const dgc_biquad_params *p, const float *x_dev, const float *cutoff_dev,
                               const float *q_dev, float *scratch_dev, float *st0, float *y_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, p && x_dev && cutoff_dev && q_dev && y_dev, "null pointer");
  int32_t rc = biquad_validate(ctx, p);
  if (rc != DGC_OK) return rc;
  const int B = p->B, T = p->T, L = p->L, NC = dgc_div_up(T, BQ_CHUNK);
  DGC_REQUIRE(ctx, NC <= 65535, "T too large");
  float *scr = scratch_dev ? scratch_dev : dgc_ctx_scratch(ctx, dgc_biquad_scratch_floats(p, 0));
  if (!scr) return DGC_ERR_OOM;
  DGC_REQUIRE(ctx, (((uintptr_t)scr) & 15) == 0, "scratch must be 16-byte aligned");
  float *coef = scr;
  double *trans = reinterpret_cast<double *>(scr + (size_t)L * 16);
  float *state = scr + ((((size_t)L * 24) + 3) & ~(size_t)3);
  // four lanes per thread when the lane count and the output alignment allow 128-bit accesses
  const bool quad = (L & 3) == 0 && L >= 16 && ((((uintptr_t)y_dev) | ((uintptr_t)state)) & 15) == 0;
  const int qx = quad ? (L / 4 >= 64 ? 64 : L / 4) : 0;
  const int nth = biquad_pairs(L), smem = biquad_stage_bytes(L);
  const dim3 grid((unsigned)(((int64_t)NC * L + nth - 1) / nth), B);
  dim3 grid4(quad ? dgc_div_up(L / 4, qx) : 1, dgc_div_up(NC, BQ4_CHUNKS), B), block4(quad ? qx : 1, BQ4_CHUNKS);
  if (!quad && smem > 48 * 1024) {
    DGC_CUDA(ctx, cudaFuncSetAttribute(biquad_fwd_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    DGC_CUDA(ctx, cudaFuncSetAttribute(biquad_fwd_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  }
  // first pass: chunk end states from a zero y-state -- as one tensor-core product when the chunks tile T exactly
  // and the problem is large enough for that path, else by running the recurrence
  const bool by_matmul = (T % BQ_CHUNK) == 0 && (double)B * NC * L >= (double)(1 << 16) && (((uintptr_t)x_dev) & 15) == 0;
  float *G = by_matmul ? state + ((((size_t)B * NC * L * 2) + 3) & ~(size_t)3) : nullptr;
  float *hist = by_matmul ? G + (size_t)L * 2 * BQ_CHUNK : nullptr;
  dgc_launch(biquad_tables_kernel, dgc_div_up(L, 4), 128, 0, ctx->stream, cutoff_dev, q_dev, L, p->gain, p->mode, coef, trans, G,
             hist);
  DGC_LAUNCHED(ctx, "biquad_tables");
  if (by_matmul) {
    rc = dgc_gemm_nt(ctx, x_dev, G, B * NC, 2 * L, BQ_CHUNK, state);
    if (rc != DGC_OK) return rc;
  } else {
    if (quad) dgc_launch(biquad_fwd4_kernel<0>, grid4, block4, 0, ctx->stream, x_dev, coef, B, T, L, NC, state, nullptr, st0);
    else dgc_launch(biquad_fwd_kernel<0>, grid, nth, smem, ctx->stream, x_dev, coef, T, L, NC, state, nullptr, st0);
    DGC_LAUNCHED(ctx, "biquad_fwd_state");
  }
  dgc_launch(biquad_carry_kernel, dim3(dgc_div_up(L, 32), B), 32, 0, ctx->stream, trans, x_dev, hist, T, L, NC,
             reinterpret_cast<float2 *>(state), st0);
  DGC_LAUNCHED(ctx, "biquad_carry");
  if (quad) dgc_launch(biquad_fwd4_kernel<1>, grid4, block4, 0, ctx->stream, x_dev, coef, B, T, L, NC, state, y_dev, st0);
  else dgc_launch(biquad_fwd_kernel<1>, grid, nth, smem, ctx->stream, x_dev, coef, T, L, NC, state, y_dev, st0);
  DGC_LAUNCHED(ctx, "biquad_fwd_out");
  if (st0) {
    dgc_launch(biquad_final_state_kernel, dgc_div_up(B * L, 128), 128, 0, ctx->stream, x_dev, y_dev, B, T, L, st0);
    DGC_LAUNCHED(ctx, "biquad_final_state");
  }
  return DGC_OK;
}

// The reverse-time pass both backward entry points share: coefficients, sweep, carry, gradients (and the loss)
template <bool UP>
static int32_t biquad_backward(dgc_ctx *ctx, const dgc_biquad_params *p, const float *x, const float *cutoff, const float *q,
                               const float *y, const float *up, float gscale, float loss_scale, float *scr, float2 *term,
                               float *gcut, float *gq, double *loss) {
  const int B = p->B, T = p->T, L = p->L, NC = dgc_div_up(T, BQ_CHUNK);
  float *coef = scr;
  float *rec = scr + ((((size_t)L * 24) + 3) & ~(size_t)3);
  const size_t rec_n = ((size_t)B * NC * BW_REC * L + 3) & ~(size_t)3;
  double *acc = reinterpret_cast<double *>(rec + rec_n);
  double *lane_loss = acc + (size_t)B * L * 6;
  dgc_launch(biquad_coef_kernel, dgc_div_up(L, 32), 32, 0, ctx->stream, cutoff, q, L, p->gain, p->mode, coef);
  DGC_LAUNCHED(ctx, "biquad_coef");
  const int nth = biquad_pairs(L), smem = biquad_stage_bytes(L);
  const dim3 grid((unsigned)(((int64_t)NC * L + nth - 1) / nth), B);
  if (smem > 48 * 1024)
    DGC_CUDA(ctx, cudaFuncSetAttribute(biquad_bwd_kernel<UP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  dgc_launch(biquad_bwd_kernel<UP>, grid, nth, smem, ctx->stream, x, coef, y, up, T, L, NC, gscale, rec);
  DGC_LAUNCHED(ctx, "biquad_bwd");
  dgc_launch(biquad_bwd_carry_kernel, dim3(dgc_div_up(L, 32), B), dim3(32, BQ_RUNS), 0, ctx->stream, rec, coef, L, NC, acc, term);
  DGC_LAUNCHED(ctx, "biquad_bwd_carry");
  dgc_launch(biquad_bwd_final_kernel, dgc_div_up(L, 8), 256, 0, ctx->stream, acc, coef, B, L, loss_scale, gcut, gq, lane_loss,
             dgc_ctx_ticket(ctx), loss);
  DGC_LAUNCHED(ctx, "biquad_bwd_final");
  return DGC_OK;
}

DGC_EXPORT int32_t dgc_biquad_mse_bwd(dgc_ctx *ctx, const dgc_biquad_params *p, const float *x_dev,
                                      const float *cutoff_dev, const float *q_dev, const float *y_dev,
                                      const float *target_dev, float loss_scale, float *scratch_dev,
                                      float *grad_cutoff_dev, float *grad_q_dev, double *loss_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, p && x_dev && cutoff_dev && q_dev && y_dev && target_dev && grad_cutoff_dev && grad_q_dev &&
                       loss_dev, "null pointer");
  int32_t rc = biquad_validate(ctx, p);
  if (rc != DGC_OK) return rc;
  DGC_REQUIRE(ctx, dgc_div_up(p->T, BQ_CHUNK) <= 65535, "T too large");
  float *scr = scratch_dev ? scratch_dev : dgc_ctx_scratch(ctx, dgc_biquad_scratch_floats(p, 1));
  if (!scr) return DGC_ERR_OOM;
  DGC_REQUIRE(ctx, (((uintptr_t)scr) & 15) == 0, "scratch must be 16-byte aligned");
  return biquad_backward<false>(ctx, p, x_dev, cutoff_dev, q_dev, y_dev, target_dev, 2.0f * loss_scale, loss_scale, scr, nullptr,
                                grad_cutoff_dev, grad_q_dev, loss_dev);
}

namespace {
// part[b][s] = sum over segment s of lam[n] * y[n-1] (n >= 1), in double
constexpr int OPG_SEGS = 32;
__global__ void __launch_bounds__(256)
onepole_ga_kernel(const float *__restrict__ lam, const float *__restrict__ y, int T, double *__restrict__ part) {
  dgc_after_previous();
  const int b = blockIdx.y, sgm = blockIdx.x;
  const int64_t per = ((int64_t)T + OPG_SEGS - 1) / OPG_SEGS, lo = max((int64_t)1, sgm * per),
                hi = min((int64_t)T, (sgm + 1) * per);
  const float *lb = lam + (size_t)b * T, *yb = y + (size_t)b * T;
  double acc = 0.0;
  for (int64_t n = lo + threadIdx.x; n < hi; n += 256) acc += (double)lb[n] * (double)yb[n - 1];
  __shared__ double sh[256];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[(size_t)b * OPG_SEGS + sgm] = sh[0];
}

__global__ void onepole_ga_sum_kernel(const double *__restrict__ part, int B, float *__restrict__ ga) {
  dgc_after_previous();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  double s = 0.0;
  for (int i = 0; i < OPG_SEGS; ++i) s += part[(size_t)b * OPG_SEGS + i];
  ga[b] = (float)s;
}
}  // namespace

// Backward of y[n] = x[n] + a y[n-1]: lam[n] = gy[n] + a lam[n+1] (the same scan, reversed in time),
// dL/dx = lam, dL/da[b] = sum_n lam[n] y[n-1].
DGC_EXPORT int32_t dgc_onepole_bwd(dgc_ctx *ctx, const float *y_dev, const float *gy_dev, int32_t B, int32_t T, float a,
                                   float *grad_x_dev, float *grad_a_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, gy_dev && grad_x_dev, "null pointer");
  DGC_REQUIRE(ctx, grad_a_dev == nullptr || y_dev != nullptr, "the coefficient gradient needs the forward output");
  DGC_REQUIRE(ctx, B > 0 && T > 0, "size out of range");
  DGC_REQUIRE(ctx, gy_dev != grad_x_dev, "in-place operation is not supported");
  DGC_REQUIRE(ctx, B <= 65535, "size out of range");
  double *part = nullptr;
  if (grad_a_dev) {
    part = reinterpret_cast<double *>(dgc_ctx_scratch(ctx, 2ull * B * OPG_SEGS));
    if (!part) return DGC_ERR_OOM;
  }
  const int32_t rc = launch_onepole<true>(ctx, gy_dev, B, T, a, nullptr, grad_x_dev, "onepole_bwd");
  if (rc != DGC_OK) return rc;
  if (grad_a_dev) {
    dgc_launch(onepole_ga_kernel, dim3(OPG_SEGS, B), 256, 0, ctx->stream, grad_x_dev, y_dev, T, part);
    DGC_LAUNCHED(ctx, "onepole_grad_a");
    dgc_launch(onepole_ga_sum_kernel, dgc_div_up(B, 128), 128, 0, ctx->stream, part, B, grad_a_dev);
    DGC_LAUNCHED(ctx, "onepole_grad_a_sum");
  }
  return DGC_OK;
}

DGC_EXPORT int32_t dgc_biquad_bwd(dgc_ctx *ctx, const dgc_biquad_params *p, const float *x_dev, const float *cutoff_dev,
                                  const float *q_dev, const float *y_dev, const float *gy_dev, float *scratch_dev,
                                  float *grad_cutoff_dev, float *grad_q_dev, float *grad_x_dev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, p && x_dev && cutoff_dev && q_dev && y_dev && gy_dev && grad_cutoff_dev && grad_q_dev,
              "null pointer");
  int32_t rc = biquad_validate(ctx, p);
  if (rc != DGC_OK) return rc;
  const int B = p->B, T = p->T, L = p->L, NC = dgc_div_up(T, BQ_CHUNK);
  DGC_REQUIRE(ctx, NC <= 65535, "T too large");
  float *scr = scratch_dev ? scratch_dev : dgc_ctx_scratch(ctx, dgc_biquad_scratch_floats(p, grad_x_dev ? 2 : 1));
  if (!scr) return DGC_ERR_OOM;
  DGC_REQUIRE(ctx, (((uintptr_t)scr) & 15) == 0, "scratch must be 16-byte aligned");
  float *after = scr + dgc_biquad_scratch_floats(p, 1);
  float2 *term = grad_x_dev ? reinterpret_cast<float2 *>(after) : nullptr;
  float *part = after + (size_t)2 * B * NC * L;
  rc = biquad_backward<true>(ctx, p, x_dev, cutoff_dev, q_dev, y_dev, gy_dev, 1.0f, 0.0f, scr, term, grad_cutoff_dev, grad_q_dev,
                             nullptr);
  if (rc != DGC_OK) return rc;
  if (grad_x_dev) {
    const dim3 grid(dgc_div_up(L, BQ_THREADS), NC, B);
    dgc_launch(biquad_gx_kernel, grid, BQ_THREADS, 0, ctx->stream, scr, gy_dev, term, B, T, L, NC, part);
    DGC_LAUNCHED(ctx, "biquad_grad_x");
    const size_t n = (size_t)B * T;
    dgc_launch(sum_partial_rows_kernel, dgc_div_up((int64_t)n, 256), 256, 0, ctx->stream, part, (int)grid.x, n, grad_x_dev);
    DGC_LAUNCHED(ctx, "biquad_grad_x_sum");
  }
  return DGC_OK;
}

// ---------------------------------------------------------------------------------------------
// One-pole filter for callers that must not allocate.
//
// A real-time audio thread (a plug-in's render callback, a driver I/O thread) may not call anything
// that allocates or may block for an unbounded time; cudaMalloc does both, and a dgc_ctx allocates
// when it is created and whenever its scratch grows.  This entry point therefore takes no context:
// the chunk-carry scratch the scan needs lives in a fixed array in device memory that is part of the
// library image (every GPU that loads the library holds these 256 KiB until the process exits), and
// the caller supplies only the stream, the input and the output.
// ---------------------------------------------------------------------------------------------
#include <atomic>
#include <mutex>

namespace {
constexpr int STATIC_MAX_CHUNKS = DGC_ONEPOLE_STATIC_MAX_CHUNKS;
// the ticket word and a cell per tile (chain.cuh)
static __device__ __align__(256) unsigned long long g_onepole_static_scratch[1 + STATIC_MAX_CHUNKS];

constexpr int STATIC_MAX_DEVICES = 64;
// Resolved device address of the array, per device.  Published once with release ordering; every later call
// reads it with one acquire load and takes no lock, so a caller on a real-time thread never waits for another
// thread that is still in its own first call on some other device.
std::mutex g_static_mutex;   // serialises the one-time look-ups only
std::atomic<unsigned long long *> g_static_ptr[STATIC_MAX_DEVICES];

void static_msg(char *buf, uint32_t len, const char *fmt, long long a = 0, long long b = 0) {
  if (buf && len) snprintf(buf, len, fmt, a, b);
}
}  // namespace

DGC_EXPORT int32_t dgc_onepole_fwd_static(void *cuda_stream, const float *x_dev, int32_t B, int32_t T, float a,
                                          float *y_dev, char *err_buf, uint32_t err_len) {
  if (err_buf && err_len) err_buf[0] = 0;
  if (!x_dev || !y_dev) {
    static_msg(err_buf, err_len, "dgc_onepole_fwd_static: null input or output pointer");
    return DGC_ERR_INVALID;
  }
  if (B <= 0 || T <= 0) {
    static_msg(err_buf, err_len, "dgc_onepole_fwd_static: B and T must be positive");
    return DGC_ERR_INVALID;
  }
  static_assert(OP_TILE == 2048, "the documented limit counts tiles");
  const long long NC = ((long long)T + 2047) / 2048;
  if ((long long)B * NC > STATIC_MAX_CHUNKS || B > 65535) {
    static_msg(err_buf, err_len,
               "dgc_onepole_fwd_static: B*ceil(T/2048) = %lld exceeds the built-in scratch of %lld chunk slots; "
               "use dgc_onepole_fwd with a context for larger signals",
               (long long)B * NC, (long long)STATIC_MAX_CHUNKS);
    return DGC_ERR_INVALID;
  }
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= STATIC_MAX_DEVICES) {
    static_msg(err_buf, err_len, "dgc_onepole_fwd_static: no usable current device (cudaGetDevice = %lld)", (long long)e);
    return DGC_ERR_CUDA;
  }
  unsigned long long *scratch = g_static_ptr[dev].load(std::memory_order_acquire);
  if (!scratch) {
    // Set-up, once per device, with that device current: the array's name is only a host-side
    // handle for the symbol; the address a kernel can use comes from cudaGetSymbolAddress.
    std::lock_guard<std::mutex> lock(g_static_mutex);
    scratch = g_static_ptr[dev].load(std::memory_order_relaxed);
    if (!scratch) {
      unsigned long long *p = nullptr;
      e = cudaGetSymbolAddress((void **)&p, g_onepole_static_scratch);
      if (e != cudaSuccess || !p) {
        static_msg(err_buf, err_len, "dgc_onepole_fwd_static: cudaGetSymbolAddress failed (%lld) on device %lld",
                   (long long)e, (long long)dev);
        return DGC_ERR_CUDA;
      }
      g_static_ptr[dev].store(p, std::memory_order_release);
      scratch = p;
    }
  }
  // an error left behind by an unrelated earlier call must not be reported as a failure of these launches
  (void)cudaGetLastError();
  cudaStream_t st = (cudaStream_t)cuda_stream;
  const int NT = (int)NC;
  const long long tiles = (long long)B * NT;
  const OnepolePowers pw = onepole_powers(a);
  if (NT > OP_REACH && pw.reach > OP_REACH) {
    onepole_passes<false>(st, x_dev, B, T, NT, pw, reinterpret_cast<float *>(scratch), nullptr, y_dev);
  } else {
    e = cudaMemsetAsync(scratch, 0, (size_t)(1 + tiles) * sizeof(*scratch), st);
    if (e != cudaSuccess) {
      static_msg(err_buf, err_len, "dgc_onepole_fwd_static: clearing the scratch failed (%lld)", (long long)e);
      return DGC_ERR_CUDA;
    }
    dgc_launch(onepole_kernel<false>, (unsigned)(tiles < 148 * OP_BLOCKS ? tiles : 148 * OP_BLOCKS), OP_THREADS, 0, st, x_dev, B,
               T, NT, pw, nullptr, y_dev, scratch, nullptr);
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    static_msg(err_buf, err_len, "dgc_onepole_fwd_static: launch failed (%lld)", (long long)e);
    return DGC_ERR_CUDA;
  }
  return DGC_OK;
}
