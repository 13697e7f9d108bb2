// fp32-accurate matmul on the 5th-generation tensor cores (tcgen05, accumulators in TMEM).
//
// C[M][N] = op(A)[M][K] * op(B)[K][N] in "3xTF32": every fp32 operand is split as x = hi + lo with hi the
// value the tensor core sees when it truncates x to TF32 and lo = x - hi (exact); the product is
// accumulated as hi*hi + hi*lo + lo*hi in fp32 in TMEM (missing term lo*lo ~ 2^-22 relative).
//
// One CTA (256 threads) owns a 128 x 128 output tile.  Per k-tile of 32 the eight warps load the fp32
// operands from global memory, split them and store hi / lo parts to shared memory in the canonical
// K-major no-swizzle layout of the UMMA shared-memory descriptor (8-row x 16-byte core matrices; rows of
// a core matrix 16 bytes apart, 8-row groups SBO apart, 16-byte k-chunks LBO apart); operands that are
// contiguous along m / n in memory are transposed on the way (vector loads, scalar stores).  One elected
// thread issues 12 tcgen05.mma (4 k-steps of 8 x 3 products) and commits them to an mbarrier; two
// shared-memory stages let the loads of tile t+1 overlap the MMAs of tile t.  The epilogue reads the
// accumulators with tcgen05.ld (32 lanes x 32 columns per warp), applies bias / tanh and stores.
// Every wait on an mbarrier is bounded: on expiry the kernel raises the status word, and still frees
// its TMEM columns before returning.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "tma.cuh"

namespace dgtc {

constexpr int TBM = 128, TBN = 128, TBK = 32, THREADS = 256;
constexpr int CHUNKS = TBK / 4;                 // 16-byte k-chunks per row
// K-major canonical layout (operand contiguous along k in memory): 16-byte unit (row r, k-chunk kc) at
// kc * LBO + r * 16; 8-row groups SBO = 128 bytes apart.
constexpr int LBO_BYTES = TBM * 16 + 16;        // k-chunk stride (one 16-byte pad against bank conflicts)
constexpr int SBO_BYTES = 8 * 16;               // 8-row group stride
// MN-major canonical layout (operand contiguous along m/n in memory): 16-byte unit = 4 consecutive m/n at one
// k, at (mn/4) * SBO_MN + (k % 8) * 16 + (k / 8) * LBO_MN (core matrix = 8 k-rows of 16 bytes, contiguous).
constexpr int SBO_MN_BYTES = 8 * 16;
constexpr int LBO_MN_BYTES = (TBM / 4) * SBO_MN_BYTES + 16;
// one operand part (hi or lo) of one stage: room for either layout
constexpr int OPER_BYTES = (CHUNKS * LBO_BYTES > (TBK / 8) * LBO_MN_BYTES) ? CHUNKS * LBO_BYTES : (TBK / 8) * LBO_MN_BYTES;
constexpr int STAGE_BYTES = 4 * OPER_BYTES;     // A_hi, A_lo, B_hi, B_lo
constexpr int SMEM_BYTES = 2 * STAGE_BYTES + 64;
constexpr uint32_t SPIN_LIMIT = 1u << 24;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

template <bool KMAJOR>
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
  // start address [0,14), leading byte offset [16,30), stride byte offset [32,46) (all >> 4),
  // descriptor version 1 at [46,48), layout type 0 (no swizzle) at [61,64)
  constexpr uint64_t lbo = KMAJOR ? LBO_BYTES : LBO_MN_BYTES, sbo = KMAJOR ? SBO_BYTES : SBO_MN_BYTES;
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((lbo >> 4) << 16) | ((sbo >> 4) << 32) | (1ull << 46);
}

// instruction descriptor: D = F32 (1 << 4), A = B = TF32 (2 << 7, 2 << 10), A / B major (0 = K, 1 = MN) at
// bits 15 / 16, N >> 3 at 17, M >> 4 at 24
template <bool A_KMAJOR, bool B_KMAJOR, int BN = TBN>
struct IDesc {
  static constexpr uint32_t value = (1u << 4) | (2u << 7) | (2u << 10) | (A_KMAJOR ? 0u : (1u << 15)) |
                                    (B_KMAJOR ? 0u : (1u << 16)) | ((uint32_t)(BN >> 3) << 17) |
                                    ((uint32_t)(TBM >> 4) << 24);
};

__device__ __forceinline__ void mma_tf32(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t IDESC, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t"
      "}\n" ::"r"(tmem_d), "l"(da), "l"(db), "r"(IDESC), "r"(accumulate), "r"(0u)
      : "memory");
}

// true in one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t"
      ".reg .pred q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t"
      "}\n"
      : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ void commit_to(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// true when the phase with the given parity has completed; bounded
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (uint32_t it = 0; it < SPIN_LIMIT; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t"
        ".reg .pred q;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t"
        "}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void split_tf32(float x, float &hi, float &lo) {
  hi = __uint_as_float(__float_as_uint(x) & 0xFFFFE000u);
  lo = x - hi;
}

// The same split with both parts ROUNDED to TF32 (round to nearest, ties away): |lo| <= 2^-11 |x| and what is
// lost, x - hi - lo, is at most 2^-22 |x| with either sign, where truncation loses up to 2^-20 |x| always
// towards zero (a bias that sums over a reduction instead of averaging out).
__device__ __forceinline__ void split_tf32_rn(float x, float &hi, float &lo) {
  // adding half a TF32 ulp to the bit pattern and clearing the 13 low bits rounds the magnitude to nearest, ties
  // away from zero (a carry into the exponent is the correct result); two integer instructions where the
  // conversion instruction runs at a quarter of their rate
  hi = __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xFFFFE000u);
  lo = __uint_as_float((__float_as_uint(x - hi) + 0x1000u) & 0xFFFFE000u);
}

// One 128 x 32 operand tile (rows r0.., k range k0..) moves in two steps so that the global loads of tile
// t+1 can be in flight while tile t is stored and multiplied: fetch() global memory -> 4 float4 registers
// per thread, stash() registers -> hi / lo parts in shared memory (256 threads).
// ROWMAJOR_K: element (r, k) at src[r * ld + k] (k contiguous): 8 lanes cover the 8 k-chunks of a row,
//   32 rows per pass, vector stores into the K-major layout.
// else: element at src[k * ld + r] (r contiguous): vector loads along m / n, transposed into the K-major
//   layout with scalar stores; a warp moves 8 k x 4 units (16 rows), a store instruction hits 8 k x 4 rows
//   with 2-way bank conflicts.  (An MN-major shared-memory descriptor with no swizzle was tried instead of
//   this transposition and produced zeros on this part, so both operands always use the K-major descriptor.)
// ROWS: 128, or 64 for the B operand of a 64-column output tile (P float4 per thread).
template <bool ROWMAJOR_K, int ROWS, int P>
__device__ __forceinline__ void fetch(const float *__restrict__ src, int ld, int rows, int r0, int k0, int k_end,
                                      int tid, float4 (&v)[P]) {
  static_assert(P == ROWS * TBK / 4 / THREADS, "a 32-deep tile, four values at a time");
  constexpr int UG = ROWS / 16, UGS = UG == 8 ? 8 : UG == 4 ? 7 : 6;   // groups of four units along the rows
  static_assert(UG == 8 || UG == 4 || UG == 2, "128, 64 or 32 rows");
  const bool vec_ok = ((ld & 3) == 0) && ((((uintptr_t)src) & 15) == 0);
#pragma unroll
  for (int p = 0; p < P; ++p) {
    v[p] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (ROWMAJOR_K) {
      const int kc = tid & 7, r = (tid >> 3) + 32 * p, gr = r0 + r, gk = k0 + 4 * kc;
      if (gr < rows) {
        const float *q = src + (size_t)gr * ld + gk;
        if (vec_ok && gk + 3 < k_end) v[p] = *reinterpret_cast<const float4 *>(q);
        else {
          if (gk < k_end) v[p].x = q[0];
          if (gk + 1 < k_end) v[p].y = q[1];
          if (gk + 2 < k_end) v[p].z = q[2];
          if (gk + 3 < k_end) v[p].w = q[3];
        }
      }
    } else {
      const int idx = p * THREADS + tid;
      const int kk = (idx & 7) + 8 * (idx >> UGS), u = ((idx >> 3) & 3) + 4 * ((idx >> 5) & (UG - 1));
      const int gk = k0 + kk, gr = r0 + 4 * u;
      if (gk < k_end) {
        const float *q = src + (size_t)gk * ld + gr;
        if (vec_ok && gr + 3 < rows) v[p] = *reinterpret_cast<const float4 *>(q);
        else {
          if (gr < rows) v[p].x = q[0];
          if (gr + 1 < rows) v[p].y = q[1];
          if (gr + 2 < rows) v[p].z = q[2];
          if (gr + 3 < rows) v[p].w = q[3];
        }
      }
    }
  }
}

template <bool ROWMAJOR_K, int ROWS, int P>
__device__ __forceinline__ void stash(const float4 (&v)[P], char *hi_part, char *lo_part, int tid) {
  constexpr int UG = ROWS / 16, UGS = UG == 8 ? 8 : UG == 4 ? 7 : 6;
#pragma unroll
  for (int p = 0; p < P; ++p) {
    if (ROWMAJOR_K) {
      const int kc = tid & 7, r = (tid >> 3) + 32 * p;
      float4 h, l;
      split_tf32(v[p].x, h.x, l.x); split_tf32(v[p].y, h.y, l.y); split_tf32(v[p].z, h.z, l.z); split_tf32(v[p].w, h.w, l.w);
      const int off = kc * LBO_BYTES + r * 16;
      *reinterpret_cast<float4 *>(hi_part + off) = h;
      *reinterpret_cast<float4 *>(lo_part + off) = l;
    } else {
      const int idx = p * THREADS + tid;
      const int kk = (idx & 7) + 8 * (idx >> UGS), u = ((idx >> 3) & 3) + 4 * ((idx >> 5) & (UG - 1));
      const float vv[4] = {v[p].x, v[p].y, v[p].z, v[p].w};
      const int base = (kk >> 2) * LBO_BYTES + (kk & 3) * 4 + (4 * u) * 16;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float h, l;
        split_tf32(vv[j], h, l);
        *reinterpret_cast<float *>(hi_part + base + j * 16) = h;
        *reinterpret_cast<float *>(lo_part + base + j * 16) = l;
      }
    }
  }
}

// tanh to ~1e-7 absolute in ~15 instructions (the library routine costs ~50 and dominated the epilogue):
// odd polynomial below 1/4 (next term 62/2835 x^9 < 1e-7 relative there), 1 - 2 / (e^{2|x|} + 1) above.
__device__ __forceinline__ float tanh_fast(float x) {
  const float ax = fabsf(x), x2 = x * x;
  const float p = x * fmaf(x2, fmaf(x2, fmaf(x2, -17.0f / 315.0f, 2.0f / 15.0f), -1.0f / 3.0f), 1.0f);
  const float e = __expf(2.0f * fminf(ax, 15.0f));
  const float t = copysignf(1.0f - __fdividef(2.0f, e + 1.0f), x);
  return ax < 0.25f ? p : t;
}

constexpr int EPI_STAGE_FLOATS = 32 * 33;   // per warp: a 32 x 32 block, rows padded to 33 floats

// Accumulators -> global memory.  Warp w may touch tensor-memory lanes 32 * (w % 4) ..; warps 0-3 take columns
// 0..63, warps 4-7 the rest; after tcgen05.ld a lane holds 32 columns of ONE output row.  Storing from there
// would make every store instruction touch 32 different rows, so each warp turns its 32 x 32 block through a
// private shared-memory tile (`stage`, EPI_STAGE_FLOATS floats per warp, the pipeline's buffers are idle by
// now) and writes full 128-byte row segments.  EPI 0: C = acc ; 1: + bias[n] ; 2: tanh(acc + bias[n]).
// Ct (optional): a second, transposed copy Ct[n][m] of the result, written straight from the registers
// (lanes = consecutive m: already 128-byte stores).
template <int EPI, int BN = TBN, int BM = TBM>
__device__ __forceinline__ void epilogue(uint32_t tmem_d, const float *__restrict__ bias, int M, int N, int m0, int n0,
                                         float *__restrict__ C, int warp, int lane, float *__restrict__ Ct,
                                         float *__restrict__ stage_all) {
  constexpr int SPAN = BN >= 64 ? BN / 2 : BN;           // columns of a warp
  const int lane_base = (warp & 3) * 32, col_base = (warp >> 2) * SPAN;
  if (lane_base >= BM || col_base >= BN) return;
  const int gm = m0 + lane_base + lane;
  float *stage = stage_all + warp * EPI_STAGE_FLOATS;
  const bool aligned = ((N & 3) == 0) && ((((uintptr_t)C) & 15) == 0);
#pragma unroll 1
  for (int c0 = col_base; c0 < col_base + SPAN; c0 += 32) {
    if (n0 + c0 >= N) break;   // the rest of this tile lies beyond the last column (warp-uniform)
    uint32_t r[32];
    const uint32_t taddr = tmem_d + ((uint32_t)lane_base << 16) + (uint32_t)c0;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    const int gn0 = n0 + c0;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      float x = __uint_as_float(r[j]);
      if (EPI >= 1 && gn0 + j < N) x += __ldg(&bias[gn0 + j]);
      if (EPI == 2) x = tanh_fast(x);
      if (Ct && gm < M && gn0 + j < N) Ct[(size_t)(gn0 + j) * M + gm] = x;
      stage[lane * 33 + j] = x;   // bank (lane + j) % 32: conflict-free
    }
    __syncwarp();
    const bool vec_ok = aligned && gn0 + 31 < N;
    if (vec_ok) {
      // 4 rows per instruction: lane -> (row it * 4 + lane / 8, columns 4 * (lane % 8) ..)
      const int rsub = lane >> 3, c4 = (lane & 7) * 4;
#pragma unroll
      for (int it = 0; it < 8; ++it) {
        const int rr = it * 4 + rsub, grow = m0 + lane_base + rr;
        const float *sp = stage + rr * 33 + c4;
        const float v0 = sp[0], v1 = sp[1], v2 = sp[2], v3 = sp[3];
        if (grow < M) *reinterpret_cast<float4 *>(C + (size_t)grow * N + gn0 + c4) = make_float4(v0, v1, v2, v3);
      }
    } else {
      // rows that are not 16-byte aligned (N not a multiple of 4) or the ragged last columns: one row per
      // instruction, lanes = consecutive columns, so every store still covers one contiguous run of a row
      const bool col_ok = gn0 + lane < N;
#pragma unroll 8
      for (int rr = 0; rr < 32; ++rr) {
        const int grow = m0 + lane_base + rr;
        const float v = stage[rr * 33 + lane];
        if (col_ok && grow < M) C[(size_t)grow * N + gn0 + lane] = v;
      }
    }
    __syncwarp();
  }
}

// A_KMAJOR: A stored [M][K]; else stored [K][M].  B_KMAJOR: B stored [N][K]; else stored [K][N].
// EPI 0: C = acc ; 1: + bias[n] ; 2: tanh(acc + bias[n]).  blockIdx.z selects a k-slice (split-K slab of C).
// BM x BN: the output tile.  Products of few tiles take smaller ones: a CTA alone on its SM waits for its own loads, 24 KB a
// k tile for 128 x 64 at the 45 bytes a cycle that one SM gets, 8 KB for 32 x 32.  The MMA stays 128 rows high (what the rows
// past BM hold goes to accumulator rows that nobody reads) and an output element adds up the same products in the same order.
// The loads run three k tiles ahead in registers, and a ninth warp issues the MMAs: from a worker, the 900 cycles that twelve
// of them and the commit take stood between two tiles of splitting and loading.
// 128 x 128 over 750 k: 51 us in one 128 x 128 tile with one k tile ahead, 38 in 128 x 64 with three, 27 in 64 x 64, 20 in
// 32 x 32; 750 x 128 over 128 k: 13 and 7.7 us.
template <bool A_KMAJOR, bool B_KMAJOR, int EPI, int BM, int BN>
__global__ void __launch_bounds__(THREADS + 32, 1)
tc_gemm_kernel(const float *__restrict__ A, const float *__restrict__ B, const float *__restrict__ bias, int M, int N,
               int K, int k_per_split, float *__restrict__ C, float *__restrict__ Ct, int32_t *status) {
  dgc_after_previous();
  extern __shared__ __align__(128) char smem[];
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + 2 * STAGE_BYTES);      // two "stage multiplied" mbarriers
  uint64_t *ready = bars + 2;                                                 // two "stage written"
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + 2 * STAGE_BYTES + 32);
  volatile int *failed = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int k_begin = blockIdx.z * k_per_split, k_end = min(K, k_begin + k_per_split);
  C += (size_t)blockIdx.z * M * N;
  const int KT = (k_end - k_begin + TBK - 1) / TBK;

  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&bars[i]), 1);
      mbar_init(smem_u32(&ready[i]), THREADS / 32);   // one arrival per worker warp
    }
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_d = *tmem_slot;

  if (warp < THREADS / 32) {
    constexpr int AHEAD = 3, PA = BM / 32, PB = BN / 32;
    float4 va[AHEAD][PA], vb[AHEAD][PB];
    auto load = [&](int kt, float4 (&fa)[PA], float4 (&fb)[PB]) {
      if (kt >= KT) return;
      fetch<A_KMAJOR, BM>(A, A_KMAJOR ? K : M, M, m0, k_begin + kt * TBK, k_end, tid, fa);
      fetch<B_KMAJOR, BN>(B, B_KMAJOR ? K : N, N, n0, k_begin + kt * TBK, k_end, tid, fb);
    };
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) load(j, va[j], vb[j]);
    auto tile = [&](int kt, float4 (&fa)[PA], float4 (&fb)[PB]) {
      const int s = kt & 1;
      // bounded; a thread that gives up raises the shared flag and everybody stops waiting
      if (kt >= 2 && !*failed && !mbar_wait(smem_u32(&bars[s]), (uint32_t)(((kt >> 1) - 1) & 1))) *failed = 1;
      char *st = smem + s * STAGE_BYTES;
      stash<A_KMAJOR, BM>(fa, st, st + OPER_BYTES, tid);
      stash<B_KMAJOR, BN>(fb, st + 2 * OPER_BYTES, st + 3 * OPER_BYTES, tid);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy writes -> async proxy (tensor core)
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ready[s]));
      load(kt + AHEAD, fa, fb);
    };
    for (int kt = 0; kt < KT; kt += AHEAD) {
#pragma unroll
      for (int j = 0; j < AHEAD; ++j)
        if (kt + j < KT) tile(kt + j, va[j], vb[j]);
    }
  } else {
    // The warp walks together and one lane issues: addresses and descriptors are then the same for the whole warp.  Worked out by
    // the one lane alone they cost about as much as its twelve MMAs.
    constexpr uint32_t ID = IDesc<true, true, BN>::value;
    const bool leader = elect_one();
    bool go = true;
    for (int kt = 0; go && kt < KT; ++kt) {
      const int s = kt & 1;
      // when the workers or the tensor core stop answering no further MMAs are issued, TMEM is still released below
      go = __all_sync(0xffffffffu, !*failed && mbar_wait(smem_u32(&ready[s]), (uint32_t)((kt >> 1) & 1)));
      if (!go) {
        *failed = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (leader) {
        const uint32_t stage = smem_u32(smem) + s * STAGE_BYTES;
        const uint64_t dah = make_desc<true>(stage), dal = make_desc<true>(stage + OPER_BYTES);
        const uint64_t dbh = make_desc<true>(stage + 2 * OPER_BYTES), dbl = make_desc<true>(stage + 3 * OPER_BYTES);
#pragma unroll
        for (int ks = 0; ks < TBK / 8; ++ks) {
          constexpr int STEP = 2 * LBO_BYTES / 16;   // 8 tf32 along k = two 16-byte k-chunks
          mma_tf32(tmem_d, dal + ks * STEP, dbh + ks * STEP, ID, (kt | ks) ? 1u : 0u);   // small terms first
          mma_tf32(tmem_d, dah + ks * STEP, dbl + ks * STEP, ID, 1u);
          mma_tf32(tmem_d, dah + ks * STEP, dbh + ks * STEP, ID, 1u);
        }
        commit_to(smem_u32(&bars[s]));
      }
      __syncwarp();
    }
    // the last commit covers every MMA issued before it
    if (KT > 0 && go && !mbar_wait(smem_u32(&bars[(KT - 1) & 1]), (uint32_t)(((KT - 1) >> 1) & 1))) *failed = 1;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  const bool ok = !*failed;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  if (ok && KT > 0) {
    if (warp < THREADS / 32) epilogue<EPI, BN, BM>(tmem_d, bias, M, N, m0, n0, C, warp, lane, Ct, reinterpret_cast<float *>(smem));
  } else if (KT == 0) {
    // empty reduction range: the slab is zero
    const int gm = m0 + (warp & 3) * 32 + lane;
    if (gm < M && warp < BM / 32)
      for (int c = 0; c < BN; ++c)
        if (n0 + c < N) C[(size_t)gm * N + n0 + c] = 0.0f;
  }
  if (!ok && tid == 0) atomicExch(status, 201);  // an MMA completion never arrived within the spin limit
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"((uint32_t)BN) : "memory");
  }
}


// ---------------------------------------------------------------------------------------------------------
// Both operands contiguous along k in memory (A [M][K], B [N][K]), rows only 4-byte aligned (K not a multiple of 4, and no pass
// before that could leave aligned copies of them): the asynchronous pipeline by 4-byte copies.  cp.async copies floats straight into the 64-byte-swizzled K-major layout (8-row groups
// of 512 bytes, 16-byte chunk c of row r at c ^ ((r / 2) % 4)), RAW raw stages deep, PF tiles ahead of the tensor core; the raw
// fp32 tile IS the "hi" operand (the tensor core reads the top 19 bits of every 32-bit word and ignores the 13 low mantissa
// bits, i.e. it truncates to TF32 itself), so the threads only compute lo = x - trunc(x), shared memory to shared memory, into
// one of two lo buffers.  Tile t's MMAs commit to an mbarrier of their own raw stage; the only wait of iteration t is on tile
// t-2 (it frees both the raw stage about to be refilled and the lo buffer about to be rewritten), two iterations after its
// MMAs were issued.  97 KB per CTA: two share an SM, and one's epilogue runs under the other's main loop.
// ---------------------------------------------------------------------------------------------------------
struct KK {
  static constexpr int BK = 16, BN = TBN, CHUNKS_K = BK / 4, ROW_BYTES = BK * 4;
  static constexpr int OPER = TBM * ROW_BYTES;            // one operand of one tile
  static constexpr int RAW = 4, PF = 2;
  static constexpr int RAW_STAGE = 2 * OPER;              // A, B
  static constexpr int SMEM = (RAW + 2) * RAW_STAGE + 128 + 1024;   // + room to align to 1024
  // byte offset of 16-byte chunk kc of row r inside one operand
  __device__ static __forceinline__ int unit_offset(int r, int kc) {
    return (r >> 3) * 512 + (r & 7) * 64 + ((kc ^ ((r >> 1) & 3)) << 4);
  }
};

// one float; src_bytes 0 = zero fill.  For operands whose rows are not 16-byte aligned (K not a multiple of 4).
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}

// K-major, 64-byte swizzle: LBO unused (1), SBO = 512 bytes between 8-row groups, layout type 4 at [61,64)
__device__ __forceinline__ uint64_t make_desc_sw64(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | ((512ull >> 4) << 32) | (1ull << 46) | (4ull << 61);
}

constexpr int KK_THREADS = THREADS + 32;   // 8 worker warps + 1 warp whose lane 0 issues the MMAs

__global__ void __launch_bounds__(KK_THREADS, 2)
tc_gemm_kk4_kernel(const float *__restrict__ A, const float *__restrict__ B, int M, int N, int K, int k_per_split,
                   float *__restrict__ C, int32_t *status) {
  dgc_after_previous();
  using G = KK;
  constexpr int BK = G::BK;
  extern __shared__ __align__(128) char smem_base[];
  // the swizzle pattern is a function of the address: tiles start on 1024-byte boundaries
  char *smem = smem_base + ((1024u - (smem_u32(smem_base) & 1023u)) & 1023u);
  char *raw = smem, *lob = smem + G::RAW * G::RAW_STAGE;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + (G::RAW + 2) * G::RAW_STAGE);  // RAW "tile consumed" mbarriers
  uint64_t *ready = bars + G::RAW;                                                    // 2 "lo buffer written" mbarriers
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + (G::RAW + 2) * G::RAW_STAGE + 64);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * TBM, n0 = blockIdx.x * TBN;
  const int k_begin = blockIdx.z * k_per_split, k_end = min(K, k_begin + k_per_split);
  C += (size_t)blockIdx.z * M * N;
  const int KT = (k_end - k_begin + BK - 1) / BK;

  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < G::RAW; ++i) mbar_init(smem_u32(&bars[i]), 1);
    mbar_init(smem_u32(&ready[0]), THREADS / 32);   // one arrival per worker warp
    mbar_init(smem_u32(&ready[1]), THREADS / 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)TBN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_d = *tmem_slot;
  bool ok = true;

  volatile int *failed = reinterpret_cast<volatile int *>(tmem_slot + 1);
  if (tid == 0) *failed = 0;
  __syncthreads();

  if (warp < THREADS / 32) {
    // ---- worker warps: copy, split, publish -----------------------------------------------------------------
    // The tile is copied float by float, element e = tid + 256 i -> (row e / BK, k = e % BK), so the lanes of a warp copy
    // consecutive floats of two rows (16-byte units would make every instruction touch eight rows).  256 % BK == 0: k is the
    // same for all of a thread's elements, its rows are 16 apart, and each element's place in shared memory moves by a constant
    // from one to the next.  The thread splits exactly the elements it copied itself, so the only synchronisation of the loop
    // is through mbarriers: "tile kt-2 consumed" before its raw stage and lo buffer are reused, "lo buffer written" towards the
    // MMA warp.
    constexpr int EPT4 = 2 * TBM * BK / THREADS;             // 16 elements per thread: 8 of A, 8 of B
    const int k4 = tid % BK, r4 = tid / BK;                  // this thread's k and first row
    const int soff4 = G::unit_offset(r4, k4 >> 2) + (k4 & 3) * 4;
    const int dsoff4 = G::unit_offset(r4 + THREADS / BK, k4 >> 2) - G::unit_offset(r4, k4 >> 2);
    auto issue_tile = [&](int kt) {
      if (kt < KT) {
        const int k0 = kt * BK;   // relative to k_begin
        const uint32_t st = smem_u32(raw + (kt % G::RAW) * G::RAW_STAGE);
        const bool kin = k_begin + k0 + k4 < k_end;
#pragma unroll
        for (int i = 0; i < EPT4; ++i) {
          const int op = i >= EPT4 / 2, r = r4 + (THREADS / BK) * (i - op * (EPT4 / 2));
          const int gr = (op ? n0 : m0) + r;
          const bool in = kin && gr < (op ? N : M);
          cp_async4(st + op * G::OPER + soff4 + (i - op * (EPT4 / 2)) * dsoff4,
                    in ? (op ? B : A) + (size_t)gr * K + k_begin + k0 + k4 : A, in ? 4 : 0);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");   // one group per call keeps the counting uniform
    };
#pragma unroll
    for (int p = 0; p < G::PF; ++p) issue_tile(p);
    for (int kt = 0; kt < KT; ++kt) {
      if (kt >= 2 && !*failed) {   // bounded; a thread that gives up raises the shared flag and everybody stops waiting
        if (!mbar_wait(smem_u32(&bars[(kt - 2) % G::RAW]), (uint32_t)(((kt - 2) / G::RAW) & 1))) *failed = 1;
      }
      issue_tile(kt + G::PF);
      asm volatile("cp.async.wait_group %0;" ::"n"(G::PF) : "memory");   // this thread's floats of tile kt landed
      char *st = raw + (kt % G::RAW) * G::RAW_STAGE, *lo = lob + (kt & 1) * G::RAW_STAGE;
      float v[EPT4];
#pragma unroll
      for (int i = 0; i < EPT4; ++i)
        v[i] = *reinterpret_cast<const float *>(st + (i >= EPT4 / 2) * G::OPER + soff4 + (i % (EPT4 / 2)) * dsoff4);
#pragma unroll
      for (int i = 0; i < EPT4; ++i) {
        float h, l;
        split_tf32(v[i], h, l);
        *reinterpret_cast<float *>(lo + (i >= EPT4 / 2) * G::OPER + soff4 + (i % (EPT4 / 2)) * dsoff4) = l;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // this thread's writes -> tensor-core proxy
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ready[kt & 1]));
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  } else {
    // ---- MMA issue: the warp walks together, one lane issues --------------------------------------------------
    constexpr uint32_t ID = IDesc<true, true>::value;
    const bool leader = elect_one();
    bool go = true;
    for (int kt = 0; go && kt < KT; ++kt) {
      go = __all_sync(0xffffffffu, !*failed && mbar_wait(smem_u32(&ready[kt & 1]), (uint32_t)((kt >> 1) & 1)));
      if (!go) {
        *failed = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (leader) {
        const uint32_t hi = smem_u32(raw) + (kt % G::RAW) * G::RAW_STAGE, lo = smem_u32(lob) + (kt & 1) * G::RAW_STAGE;
        const uint64_t dah = make_desc_sw64(hi), dbh = make_desc_sw64(hi + G::OPER);
        const uint64_t dal = make_desc_sw64(lo), dbl = make_desc_sw64(lo + G::OPER);
#pragma unroll
        for (int ks = 0; ks < BK / 8; ++ks) {   // 8 tf32 along k: 32 bytes further inside the swizzled row
          mma_tf32(tmem_d, dal + ks * 2, dbh + ks * 2, ID, (kt | ks) ? 1u : 0u);
          mma_tf32(tmem_d, dah + ks * 2, dbl + ks * 2, ID, 1u);
          mma_tf32(tmem_d, dah + ks * 2, dbh + ks * 2, ID, 1u);
        }
        commit_to(smem_u32(&bars[kt % G::RAW]));
      }
      __syncwarp();
    }
    // the last commit covers every MMA issued before it
    if (KT > 0 && go && !mbar_wait(smem_u32(&bars[(KT - 1) % G::RAW]), (uint32_t)(((KT - 1) / G::RAW) & 1))) *failed = 1;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  ok = !*failed;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  if (ok && KT > 0) {
    if (warp < THREADS / 32) epilogue<0>(tmem_d, nullptr, M, N, m0, n0, C, warp, lane, nullptr, reinterpret_cast<float *>(smem));
  } else if (KT == 0) {
    const int gm = m0 + (warp & 3) * 32 + lane;
    if (gm < M && warp < 4)
      for (int c = 0; c < TBN; ++c)
        if (n0 + c < N) C[(size_t)gm * N + n0 + c] = 0.0f;
  }
  if (!ok && tid == 0) atomicExch(status, 201);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"((uint32_t)TBN) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------------------
// Both operands contiguous along k, 16-byte aligned rows: operand A in tensor memory, one persistent CTA per
// SM.  Fetching both operands from shared memory for each of the three products, a pipeline like the one above carries 96 KB of
// it per 16 k of a 128 x 128 tile, 768 cycles for 384 of multiplying, and a CTA's split, products and epilogue come one
// after the other.  Here
//   load      one thread has the copy engine bring 64-byte-swizzled tiles of both operands, RAW of them ahead
//   split     eight warps in two groups, a tile each in turn: a group's lanes are the rows of A, whose hi and lo parts go to
//             tensor memory side by side, a column per k; B's lo part goes to shared memory, its hi part is the raw tile
//   multiply  one warp; the MMAs fetch only B from shared memory (64 KB in all) and fill one of two accumulators
//   store     eight warps move the other accumulator, of the tile before, to global memory
// The products and the order of their sums are those of a pipeline with both operands in shared memory: the same bits.
// Bound by the shared memory, 512 cycles a tile (525 measured; the multiplying alone 393).  32000 x 512 over 512 k with
// tanh, 16-byte copies and both operands in shared memory: 144 us; A in tensor memory, two CTAs per SM: 128, with two groups of
// splitting warps (800 cycles from a tile's arrival to its split) 112; persistent with the epilogue apart 111, with the issuing
// warp walking together 84.  Three or four groups: 88.  512 x 512 over 32000 k in 18 slices: 99 -> 80.
// The 128 x 256 tiles of a long reduction have one accumulator: there is one tile for a CTA.
// ---------------------------------------------------------------------------------------------------------
template <int BN>
struct TS {
  static constexpr int BK = 16, ROW_BYTES = BK * 4, RAW = BN == 128 ? 8 : 4, ACCS = BN == 128 ? 2 : 1;
  static constexpr int A_BYTES = TBM * ROW_BYTES, B_BYTES = BN * ROW_BYTES, STAGE = A_BYTES + B_BYTES;
  static constexpr int GROUPS = 2, SPLITTERS = 4 * GROUPS, STORERS = 8;          // warps
  static constexpr int THREADS_ALL = 32 * (SPLITTERS + STORERS + 2);
  static constexpr int OFF_LO = RAW * STAGE, OFF_EPI = OFF_LO + RAW * B_BYTES, OFF_BARS = OFF_EPI + STORERS * EPI_STAGE_FLOATS * 4;
  static constexpr int SMEM = OFF_BARS + 256 + 1024;             // + room to align to 1024
  static constexpr int COLS = 512;                               // tensor memory: accumulators, split stages of A
};
static_assert(TS<128>::SMEM <= 227 * 1024 && TS<256>::SMEM <= 227 * 1024, "shared memory of one CTA");
static_assert(2 * 128 + TS<128>::RAW * 32 <= 512 && 256 + TS<256>::RAW * 32 <= 512, "tensor memory");

// the same wait for one of several that give up together: who runs out raises the flag, who sees it raised stops waiting
__device__ __forceinline__ bool mbar_wait_or(uint32_t bar, uint32_t parity, volatile int *failed) {
  for (uint32_t it = 0; it < SPIN_LIMIT; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t"
        ".reg .pred q;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t"
        "}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 255u) == 255u && *failed) return false;
  }
  *failed = 1;
  return false;
}

__device__ __forceinline__ void mma_tf32_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t IDESC, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t"
      "}\n" ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(IDESC), "r"(accumulate), "r"(0u)
      : "memory");
}

__device__ __forceinline__ void tmem_store8(uint32_t taddr, const float (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "f"(v[0]), "f"(v[1]),
               "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

template <int EPI, int BN>
__global__ void __launch_bounds__(TS<BN>::THREADS_ALL, 1)
tc_gemm_ts_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  const float *__restrict__ bias, int M, int N, int K, int k_per_split, int items, float *__restrict__ C,
                  float *__restrict__ Ct, int32_t *status) {
  dgc_after_previous();
  using G = TS<BN>;
  extern __shared__ __align__(128) char smem_base[];
  char *smem = smem_base + ((1024u - (smem_u32(smem_base) & 1023u)) & 1023u);   // the swizzle is a function of the address
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + G::OFF_BARS);   // raw tile landed
  uint64_t *ready = full + G::RAW;                                     // split written
  uint64_t *consumed = ready + G::RAW;                                 // multiplied
  uint64_t *summed = consumed + G::RAW;                                // accumulator complete
  uint64_t *stored = summed + G::ACCS;                                 // accumulator read
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(stored + G::ACCS);
  volatile int *failed = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < G::RAW; ++i) {
      mbar_init(smem_u32(&full[i]), 1);
      mbar_init(smem_u32(&ready[i]), 4);   // one arrival per warp of a group
      mbar_init(smem_u32(&consumed[i]), 1);
    }
#pragma unroll
    for (int i = 0; i < G::ACCS; ++i) {
      mbar_init(smem_u32(&summed[i]), 1);
      mbar_init(smem_u32(&stored[i]), G::STORERS);
    }
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)G::COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_d = *tmem_slot, tmem_a = tmem_d + G::ACCS * BN;

  // item: (k slice, row tile, column tile), column tiles next to each other; this CTA takes every gridDim.x-th
  const int nx = (N + BN - 1) / BN, ny = (M + TBM - 1) / TBM;
  struct Item {
    int m0, n0, k0, z, tiles;
  };
  auto item_at = [&](int i) {
    Item t;
    t.n0 = i % nx * BN;
    t.m0 = i / nx % ny * TBM;
    t.z = i / nx / ny;
    t.k0 = t.z * k_per_split;
    t.tiles = (min(K, t.k0 + k_per_split) - t.k0 + G::BK - 1) / G::BK;
    return t;
  };
  // g: k tiles counted through all items; a: items of this CTA
  auto wait = [&](uint64_t *bars, int g) {
    return mbar_wait_or(smem_u32(&bars[g % G::RAW]), (uint32_t)((g / G::RAW) & 1), failed);
  };
  auto wait_acc = [&](uint64_t *bars, int a) {
    return mbar_wait_or(smem_u32(&bars[a % G::ACCS]), (uint32_t)((a / G::ACCS) & 1), failed);
  };
  if (warp < G::SPLITTERS) {
    // ---- split: row 32 (warp % 4) + lane of A, 16-byte units of B -------------------------------------------
    const int gtid = tid & 127, r = gtid, row_off = (r >> 3) * 512 + (r & 7) * 64, swz = (r >> 1) & 3;
    const uint32_t a_dst = tmem_a + ((uint32_t)((warp & 3) * 32) << 16);
    constexpr int UPT = BN * G::BK / 4 / 128;
    int total = 0;
    for (int i = blockIdx.x; i < items; i += gridDim.x) total += item_at(i).tiles;
    for (int g = warp >> 2; g < total; g += G::GROUPS) {
      const int s = g % G::RAW;
      // landed, and the split stage free (the loader waited for that, too); the whole warp goes on or gives up
      const bool go = wait(full, g) && (g < G::RAW || wait(consumed, g - G::RAW));
      if (!__all_sync(0xffffffffu, go)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const char *st = smem + s * G::STAGE;
      float4 u[4], v[UPT];
#pragma unroll
      for (int i = 0; i < 4; ++i) u[i] = *reinterpret_cast<const float4 *>(st + row_off + ((i ^ swz) << 4));
#pragma unroll
      for (int i = 0; i < UPT; ++i) v[i] = *reinterpret_cast<const float4 *>(st + G::A_BYTES + (gtid + 128 * i) * 16);
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        const float x[8] = {u[i].x, u[i].y, u[i].z, u[i].w, u[i + 1].x, u[i + 1].y, u[i + 1].z, u[i + 1].w};
        float h[8], l[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) split_tf32(x[j], h[j], l[j]);
        tmem_store8(a_dst + s * 2 * G::BK + 4 * i, h);
        tmem_store8(a_dst + s * 2 * G::BK + G::BK + 4 * i, l);
      }
      char *lo = smem + G::OFF_LO + s * G::B_BYTES;
#pragma unroll
      for (int i = 0; i < UPT; ++i) {
        float4 hh, ll;
        split_tf32(v[i].x, hh.x, ll.x); split_tf32(v[i].y, hh.y, ll.y); split_tf32(v[i].z, hh.z, ll.z); split_tf32(v[i].w, hh.w, ll.w);
        *reinterpret_cast<float4 *>(lo + (gtid + 128 * i) * 16) = ll;   // the same place in the same swizzle
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // this thread's writes -> tensor-core proxy
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ready[s]));
    }
  } else if (warp < G::SPLITTERS + G::STORERS) {
    // ---- store ----------------------------------------------------------------------------------------------
    const int w = warp - G::SPLITTERS;
    int a = 0;
    for (int i = blockIdx.x; i < items; i += gridDim.x, ++a) {
      if (!__all_sync(0xffffffffu, wait_acc(summed, a))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const Item t = item_at(i);
      epilogue<EPI, BN>(tmem_d + a % G::ACCS * BN, bias, M, N, t.m0, t.n0, C + (size_t)t.z * M * N, w, lane, Ct,
                        reinterpret_cast<float *>(smem + G::OFF_EPI));
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&stored[a % G::ACCS]));
    }
  } else if (warp == G::SPLITTERS + G::STORERS) {
    // ---- multiply: the warp walks together, one lane issues ---------------------------------------------------
    // (so that stages, addresses and descriptors are the same for the whole warp: worked out by the one lane alone, they and
    // the six MMAs took 610 cycles a tile)
    constexpr uint32_t ID = IDesc<true, true, BN>::value;
    const bool leader = elect_one();
    const uint32_t raw0 = smem_u32(smem), lo0 = raw0 + G::OFF_LO;
    int a = 0, s = 0, phase = 0;
    bool go = true;
    for (int i = blockIdx.x; go && i < items; i += gridDim.x, ++a) {
      go = __all_sync(0xffffffffu, a < G::ACCS || wait_acc(stored, a - G::ACCS));
      const int tiles = item_at(i).tiles;
      const uint32_t acc = tmem_d + a % G::ACCS * BN;
      for (int k = 0; go && k < tiles; ++k) {
        go = __all_sync(0xffffffffu, mbar_wait_or(smem_u32(&ready[s]), phase, failed));
        if (!go) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (leader) {
          const uint64_t bh = make_desc_sw64(raw0 + s * G::STAGE + G::A_BYTES);
          const uint64_t bl = make_desc_sw64(lo0 + s * G::B_BYTES);
          const uint32_t a_hi = tmem_a + s * 2 * G::BK, a_lo = a_hi + G::BK;
#pragma unroll
          for (int ks = 0; ks < G::BK / 8; ++ks) {   // 8 k: 32 bytes further inside the swizzled row, 8 columns
            mma_tf32_ts(acc, a_lo + ks * 8, bh + ks * 2, ID, k | ks ? 1u : 0u);
            mma_tf32_ts(acc, a_hi + ks * 8, bl + ks * 2, ID, 1u);
            mma_tf32_ts(acc, a_hi + ks * 8, bh + ks * 2, ID, 1u);
          }
          commit_to(smem_u32(&consumed[s]));
          if (k == tiles - 1) commit_to(smem_u32(&summed[a % G::ACCS]));   // covers every MMA issued before it
        }
        __syncwarp();
        if (++s == G::RAW) {
          s = 0;
          phase ^= 1;
        }
      }
    }
    if (go && a > 0) wait_acc(summed, a - 1);
  } else if (lane == 0) {
    // ---- load -----------------------------------------------------------------------------------------------
    int g = 0;
    bool go = true;
    for (int i = blockIdx.x; go && i < items; i += gridDim.x) {
      const Item t = item_at(i);
      for (int k = 0; k < t.tiles; ++k, ++g) {
        go = g < G::RAW || wait(consumed, g - G::RAW);
        if (!go) break;
        char *st = smem + g % G::RAW * G::STAGE;
        uint64_t *bar = &full[g % G::RAW];
        dgtma::mbar_expect_tx(bar, G::STAGE);
        dgtma::load_2d(st, &map_a, t.k0 + k * G::BK, t.m0, bar);
        dgtma::load_2d(st + G::A_BYTES, &map_b, t.k0 + k * G::BK, t.n0, bar);
      }
    }
    for (int i = max(0, g - G::RAW); i < g; ++i)   // nothing of this block's is in flight when it ends
      if (!mbar_wait(smem_u32(&full[i % G::RAW]), (uint32_t)((i / G::RAW) & 1))) *failed = 1;
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*failed && tid == 0) atomicExch(status, 201);
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"((uint32_t)G::COLS) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------------------
// Short reductions (K <= 72; the band -> tap map has K = 65, N = 257): A [M][K], B [N][K], both contiguous
// along k.  With so few k-tiles a CTA per output tile spends its life in prologue, load latency and epilogue,
// so this kernel is persistent: a CTA owns ONE 128-column block of the output, keeps that block of B (hi and
// lo parts) in shared memory for its whole life and walks down the row tiles of A.
//   copy     a 128-row tile of A is one contiguous, 16-byte aligned run of 128 K floats whatever K's alignment:
//            the thread that issues the MMAs fetches it with ONE bulk copy (cp.async.bulk, completion on an
//            mbarrier) into a linear staging buffer, as soon as the previous tile has been split out of it
//   split    sixteen worker warps read the linear tile and write its hi and lo parts (both rounded to TF32) into
//            the K-major no-swizzle layout of make_desc<true>(): 16-byte unit (row r, chunk kc) at
//            kc * LBO_BYTES + r * 16; k is padded to a multiple of 8 with zeros that are written once
//   multiply one thread issues the 3 x ceil(K / 8) MMAs of the tile into one of TWO 128-column accumulators
//   store    while the tensor core works on tile i, the worker warps move tile i-1 from the other accumulator to
//            global memory (32 x 16 blocks turned through shared memory into 64-byte row segments)
// N % 128 <= SK::EXTRA_MAX leftover columns (the 257th tap) are plain fp32 dot products of the CTAs of the
// last column block, from the linear tile, instead of a third block of 127 empty columns.
// Every wait is bounded; on expiry the kernel raises status 202, stops waiting everywhere and frees its TMEM.
// ---------------------------------------------------------------------------------------------------------
struct SK {
  static constexpr int KP_MAX = 72;                          // largest K (nine k-steps of 8)
  static constexpr int WORKERS = 512, THREADS_ALL = WORKERS + 32;
  static constexpr int OPER = (KP_MAX / 4) * LBO_BYTES;      // one operand part: 18 chunks
  static constexpr int OFF_BHI = 0, OFF_BLO = OPER, OFF_AHI = 2 * OPER, OFF_ALO = 3 * OPER, OFF_LIN = 4 * OPER;
  static constexpr int LIN_BYTES = TBM * KP_MAX * 4;
  static constexpr int EPI_ROW = 20;                         // floats per staged row of 16 (16-byte stores, no conflicts)
  static constexpr int OFF_STAGE = OFF_LIN + LIN_BYTES;
  static constexpr int OFF_BARS = OFF_STAGE + (WORKERS / 32) * 32 * EPI_ROW * 4;
  static constexpr int SMEM = OFF_BARS + 64;
  static constexpr int EPT = TBM * KP_MAX / WORKERS;         // elements of a tile per worker thread
  static constexpr int EXTRA_MAX = 8;
};
static_assert(SK::SMEM <= 227 * 1024, "the persistent small-K kernel must fit one CTA's shared memory");
static_assert(SK::OFF_LIN % 128 == 0 && SK::OFF_STAGE % 16 == 0 && SK::OFF_BARS % 8 == 0, "alignment of the buffers");

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// linear global -> shared copy by the copy engine; both addresses 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__global__ void __launch_bounds__(SK::THREADS_ALL, 1)
tc_gemm_smallk_kernel(const float *__restrict__ A, const float *__restrict__ B, int M, int N, int K, int nblk,
                      int n_extra, int ctas_per_blk, float *__restrict__ C, int32_t *status) {
  dgc_after_previous();
  extern __shared__ __align__(128) char smem[];
  char *b_hi = smem + SK::OFF_BHI, *b_lo = smem + SK::OFF_BLO, *a_hi = smem + SK::OFF_AHI, *a_lo = smem + SK::OFF_ALO;
  float *lin = reinterpret_cast<float *>(smem + SK::OFF_LIN);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + SK::OFF_BARS);
  const uint32_t bar_ready = smem_u32(bars), bar_done = smem_u32(bars + 1), bar_load = smem_u32(bars + 2);
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + SK::OFF_BARS + 32);
  volatile int *failed = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cb = blockIdx.x % nblk, slot = blockIdx.x / nblk;
  const int n0 = cb * TBN;
  const int row_tiles = (M + TBM - 1) / TBM;
  const int nt = (row_tiles - slot + ctas_per_blk - 1) / ctas_per_blk;   // row tiles slot, slot + ctas_per_blk, ...
  const bool has_extra = n_extra > 0 && cb == nblk - 1;
  const int ksteps = (K + 7) / 8;
  const int tile_elems = TBM * K;

  // zeros once: the k padding of all four operand parts and the rows past the end of B are never written again
  for (int u = tid; u < SK::OFF_LIN / 16; u += SK::THREADS_ALL)
    reinterpret_cast<float4 *>(smem)[u] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (tid == 0) {
    mbar_init(bar_ready, SK::WORKERS / 32);   // one arrival per worker warp
    mbar_init(bar_done, 1);
    mbar_init(bar_load, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *failed = 0;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)(2 * TBN))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_d = *tmem_slot;

  if (warp < SK::WORKERS / 32) {
    // ---- worker warps ---------------------------------------------------------------------------------------
    // element e = tid + 512 j of a tile is (row e / K, k = e % K); its byte offset inside an operand part is the
    // same for A and B and fixed for the life of the thread
    unsigned short off[SK::EPT];
    {
      int r = tid / K, k = tid - r * K;
      const int dr = SK::WORKERS / K, dk = SK::WORKERS - dr * K;
#pragma unroll
      for (int j = 0; j < SK::EPT; ++j) {
        off[j] = (unsigned short)((k >> 2) * LBO_BYTES + r * 16 + (k & 3) * 4);   // < 65536 (rows past 127: unused)
        r += dr; k += dk;
        if (k >= K) { k -= K; ++r; }
      }
    }
    // this CTA's block of B, split once
    {
      const size_t b0 = (size_t)n0 * K, bend = (size_t)N * K;
#pragma unroll
      for (int j = 0; j < SK::EPT; ++j) {
        const int e = tid + SK::WORKERS * j;
        if (e < tile_elems && b0 + e < bend) {
          float h, l;
          split_tf32_rn(__ldg(B + b0 + e), h, l);
          *reinterpret_cast<float *>(b_hi + off[j]) = h;
          *reinterpret_cast<float *>(b_lo + off[j]) = l;
        }
      }
    }
    // accumulator i & 1 -> C, after the MMAs of tile i completed.  Warp w may read tensor-memory lanes
    // 32 (w % 4) ..; it takes columns 32 (w / 4) .. of them, sixteen at a time: after tcgen05.ld a lane holds 16
    // columns of ONE row, the block is turned through the warp's private staging rows, and every store
    // instruction writes two 64-byte row segments.
    float *stage = reinterpret_cast<float *>(smem + SK::OFF_STAGE) + warp * 32 * SK::EPI_ROW;
    auto store_tile = [&](int i) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int lane_base = (warp & 3) * 32, m0 = (slot + i * ctas_per_blk) * TBM;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c0 = (warp >> 2) * 32 + 16 * h, gn0 = n0 + c0;
        if (gn0 >= N) break;   // warp-uniform: the rest of this block lies beyond the last column
        uint32_t r[16];
        const uint32_t taddr = tmem_d + (uint32_t)((i & 1) * TBN) + ((uint32_t)lane_base << 16) + (uint32_t)c0;
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int q = 0; q < 4; ++q)
          *reinterpret_cast<uint4 *>(stage + lane * SK::EPI_ROW + 4 * q) = make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
        __syncwarp();
        // an instruction stores rows r and r + 4: 4 x 20 floats apart, i.e. 16 banks apart, so the two 16-float
        // segments it reads from the staging rows cover all 32 banks once
        const int rsub = lane >> 4, col = lane & 15;
        const bool col_ok = gn0 + col < N;
        float v[16];
#pragma unroll
        for (int it = 0; it < 16; ++it) v[it] = stage[((it & 3) + 8 * (it >> 2) + 4 * rsub) * SK::EPI_ROW + col];
#pragma unroll
        for (int it = 0; it < 16; ++it) {
          const int grow = m0 + lane_base + (it & 3) + 8 * (it >> 2) + 4 * rsub;
          if (col_ok && grow < M) C[(size_t)grow * N + gn0 + col] = v[it];
        }
        __syncwarp();
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    };
    for (int i = 0; i < nt; ++i) {
      // tile i has landed in the linear buffer; tile i-1 is multiplied: its accumulator is complete and the
      // operand parts of A may be overwritten
      if (!*failed && !mbar_wait(bar_load, (uint32_t)(i & 1))) *failed = 1;
      if (i >= 1 && !*failed && !mbar_wait(bar_done, (uint32_t)((i - 1) & 1))) *failed = 1;
      if (has_extra) {
        // four threads per row, every fourth k each (all loads first, then one chain of multiply-adds), combined in
        // a fixed order
        const int r = tid >> 2, part = tid & 3, gm = (slot + i * ctas_per_blk) * TBM + r;
        const float *ar = lin + r * K + part;
        for (int x = 0; x < n_extra; ++x) {
          const float *bx = B + (size_t)(nblk * TBN + x) * K + part;
          float av[SK::KP_MAX / 4], bv[SK::KP_MAX / 4];
#pragma unroll
          for (int m = 0; m < SK::KP_MAX / 4; ++m) {
            const bool in = 4 * m + part < K;
            av[m] = in ? ar[4 * m] : 0.0f;
            bv[m] = in ? __ldg(bx + 4 * m) : 0.0f;
          }
          float acc = 0.0f;
#pragma unroll
          for (int m = 0; m < SK::KP_MAX / 4; ++m) acc = fmaf(av[m], bv[m], acc);
          acc += __shfl_xor_sync(0xffffffffu, acc, 1);
          acc += __shfl_xor_sync(0xffffffffu, acc, 2);
          if (part == 0 && gm < M) C[(size_t)gm * N + nblk * TBN + x] = acc;
        }
      }
      {
        float v[SK::EPT];
#pragma unroll
        for (int j = 0; j < SK::EPT; ++j) {
          const int e = tid + SK::WORKERS * j;
          v[j] = e < tile_elems ? lin[e] : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < SK::EPT; ++j) {
          const int e = tid + SK::WORKERS * j;
          if (e < tile_elems) {
            float h, l;
            split_tf32_rn(v[j], h, l);
            *reinterpret_cast<float *>(a_hi + off[j]) = h;
            *reinterpret_cast<float *>(a_lo + off[j]) = l;
          }
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // this thread's writes -> tensor-core proxy
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_ready);
      if (i >= 1 && !*failed) store_tile(i - 1);   // while the tensor core multiplies tile i
    }
    if (nt > 0 && !*failed && !mbar_wait(bar_done, (uint32_t)((nt - 1) & 1))) *failed = 1;
    if (nt > 0 && !*failed) store_tile(nt - 1);
  } else {
    // ---- copy and MMA issue: the warp walks together, one lane issues -----------------------------------------
    constexpr uint32_t ID = IDesc<true, true, TBN>::value;
    const bool leader = elect_one();
    auto load_tile = [&](int i) {   // the CTA's i-th row tile -> linear buffer (rows past M keep stale values: never stored)
      const size_t a0 = (size_t)(slot + i * ctas_per_blk) * TBM * K, aend = (size_t)M * K;
      const size_t left = aend - a0;
      const uint32_t elems = left < (size_t)tile_elems ? (uint32_t)left : (uint32_t)tile_elems;
      const uint32_t bulk = (elems * 4u) & ~15u;
      for (uint32_t e = bulk / 4; e < elems; ++e) lin[e] = A[a0 + e];   // at most three floats of a ragged last tile
      mbar_expect_tx(bar_load, bulk);   // (release: the plain stores above are visible to whoever sees the phase)
      bulk_load(smem_u32(lin), A + a0, bulk, bar_load);
    };
    if (nt > 0 && leader) load_tile(0);
    for (int i = 0; i < nt; ++i) {
      if (!__all_sync(0xffffffffu, !*failed && mbar_wait(bar_ready, (uint32_t)(i & 1)))) {
        *failed = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (leader) {
        if (i + 1 < nt) load_tile(i + 1);   // every worker has read tile i out of the linear buffer
        const uint32_t d = tmem_d + (uint32_t)((i & 1) * TBN), s0 = smem_u32(smem);
        uint64_t dah = make_desc<true>(s0 + SK::OFF_AHI), dal = make_desc<true>(s0 + SK::OFF_ALO);
        uint64_t dbh = make_desc<true>(s0 + SK::OFF_BHI), dbl = make_desc<true>(s0 + SK::OFF_BLO);
        for (int ks = 0; ks < ksteps; ++ks) {
          mma_tf32(d, dal, dbh, ID, ks ? 1u : 0u);
          mma_tf32(d, dah, dbl, ID, 1u);
          mma_tf32(d, dah, dbh, ID, 1u);
          constexpr int STEP = 2 * LBO_BYTES / 16;   // 8 tf32 along k: two 16-byte chunks
          dah += STEP, dal += STEP, dbh += STEP, dbl += STEP;
        }
        commit_to(bar_done);
      }
      __syncwarp();
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*failed && tid == 0) atomicExch(status, 202);
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"((uint32_t)(2 * TBN)) : "memory");
  }
}

}  // namespace dgtc
