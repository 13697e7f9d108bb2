// Shared declarations of libdgen_cuda: context object, error plumbing, launch helpers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <map>
#include <string>
#include <utility>

#include "../../include/dgen_cuda.h"

#define DGC_EXPORT extern "C" __attribute__((visibility("default")))

// upload events of a host-buffer step: harmonic controls, noise branch, then one per group of voices of the target
constexpr int DGC_COPY_EVENTS = 2 + 4;

struct dgc_ctx {
  int device = 0;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev_begin = nullptr, ev_end = nullptr, ev_sync = nullptr;
  int32_t *status_dev = nullptr;  // device status word: kernels report failures here
  // cells of launches whose blocks hand values on (chain.cuh): one set for the context stream, one for the side stream,
  // so that a plan may run such a launch on both at once
  unsigned long long *chain_dev[2] = {nullptr, nullptr};
  uint64_t chain_cells[2] = {0, 0};
  // last-block-done counters of the multi-block reductions (kept at 0), one for the context stream and one for the side
  // stream: a plan may reduce on both at once (dgc_ctx_ticket)
  unsigned int *ticket_dev = nullptr;
  int64_t launches = 0;
  char err[512] = {0};
  int sm_count = 148;
  // context-owned scratch (grown on demand, never shrunk), one for the context stream and one for the side stream
  float *scratch[2] = {nullptr, nullptr};
  uint64_t scratch_floats[2] = {0, 0};
  // bumped whenever a context-owned device buffer (scratch, staging, transposed-operand copies) is freed or
  // reallocated: a recorded step holds raw pointers into those buffers and must be re-recorded afterwards
  uint64_t buffer_generation = 0;
  // cached data-independent tables
  std::map<std::pair<int, int>, float *> playheads;  // (F, T) -> device clock
  std::map<std::pair<int, int>, int *> row_ranges;   // (F, T) -> [F][4] frame ranges per control row
  std::map<std::pair<int, int>, float2 *> row_tables;  // (F, T) -> per frame (floor row as int bits, fraction)
  std::map<int, float *> hann_sym;                   // N -> symmetric Hann (spectral loss)
  std::map<int, float *> hann_per;                   // N -> periodic Hann (hann())
  std::map<int, float2 *> twiddles;                  // N -> exp(-2 pi i m / N), m < N
  double *loss_accum = nullptr;                      // 512 doubles: [0..64) results, [64..320) per-block sums
  float *wt_buf = nullptr;  // transposed copy of the current layer's weights (matmul forward)
  uint64_t wt_floats = 0;
  float *dzt_buf = nullptr;  // transposed copy of the current layer's output gradient (matmul backward)
  uint64_t dzt_floats = 0;
  uint64_t dzt_refused = UINT64_MAX;       // floats that once found no room there: not asked for again
  // staging for the host-buffer composite entry points; uploads run on their own stream so that the
  // first kernels start while later inputs are still crossing PCIe
  cudaStream_t aux_stream = nullptr;   // second stream of the composite steps (noise branch beside the harmonic one)
  cudaEvent_t fork_ev = nullptr, join_ev = nullptr;
  cudaStream_t copy_stream = nullptr;
  cudaEvent_t copy_ev[DGC_COPY_EVENTS] = {};
  cudaStream_t out_stream = nullptr;   // results on their way to the host while the step goes on
  cudaEvent_t audio_ev = nullptr, out_ev = nullptr;
  // small inputs are gathered here and cross PCIe as one copy: the blocking call's block and one per step in flight
  float *pinned[3] = {nullptr, nullptr, nullptr};
  uint64_t pinned_floats[3] = {0, 0, 0};
  int32_t *status_host = nullptr;      // page-locked copy of the status word
  float *stage_dev = nullptr;
  uint64_t stage_floats = 0;
  // two host-buffer steps in flight (plans.cu): per-slot input staging, upload events, end-of-step event
  float *pipe_in[2] = {nullptr, nullptr};
  uint64_t pipe_in_floats[2] = {0, 0};
  cudaEvent_t pipe_ev[2][DGC_COPY_EVENTS] = {};
  cudaEvent_t pipe_done[2] = {nullptr, nullptr};
  bool pipe_used[2] = {false, false}, pipe_pending[2] = {false, false};
  // NCCL communicator of the gradient exchange (comm.cu); nullptr = a world of one
  void *comm = nullptr;
  int comm_world = 1;
  // spectral-loss backward: windows owned per block, chosen per (N, hop, H, B) so that the grid fills whole waves
  std::map<std::pair<std::pair<int, int>, std::pair<int, int>>, int> mss_bwd_owned;
  // matrix products issued per kernel family since the context was created (dgc_gemm_path_counts):
  // 0 SIMT register tiles, 1 tcgen05 generic-orientation kernel, 2 tcgen05 asynchronous pipeline, 3 the same with 128 x 256 tiles
  int64_t gemm_paths[4] = {0, 0, 0, 0};
  // step recording (graph.cu)
  bool capturing = false;
  cudaStream_t capture_stream = nullptr;   // the stream the recording started on (calls inside may rebind the context)
  int64_t capture_launches0 = 0;
};

// the caller-owned flat float arena (device memory) of dgc_arena_create
struct dgc_arena {
  dgc_ctx *ctx;
  float *ptr;
  uint64_t n;
  bool owned = true;   // false: the memory belongs to the caller (dgc_arena_wrap)
};

int32_t dgc_fail(dgc_ctx *ctx, int32_t code, const char *fmt, ...);
int32_t dgc_check_launch(dgc_ctx *ctx, const char *what);
// DGC_ERR_DEVICE (the word is cleared) when a kernel left something in the status word
int32_t dgc_report_status(dgc_ctx *ctx, int32_t status);
// returns device pointer to at least n floats of the current stream's context scratch (nullptr + error set on failure)
float *dgc_ctx_scratch(dgc_ctx *ctx, uint64_t nfloats);
// 1 + n 64-bit words for ONE launch on the current stream, cleared there: the ticket word, then n cells (chain.cuh)
unsigned long long *dgc_ctx_chain(dgc_ctx *ctx, uint64_t n);
// [F][4] ints: frames whose floor control row is r are [a,b) and [c,d) (second run: after the clock wrap)
const int *dgc_ctx_row_ranges(dgc_ctx *ctx, int F, int T);
// [T] float2: x = bits of the floor control row (int), y = lerp fraction of sampleRow at the cached clock
const float2 *dgc_ctx_row_table(dgc_ctx *ctx, int F, int T);
// N values, then the same N turned by one place (the last one first)
const float *dgc_ctx_hann_sym(dgc_ctx *ctx, int N);
const float *dgc_ctx_hann_per(dgc_ctx *ctx, int N);
// C[M][N] = A[M][K] * B[N][K]^T on the matmul path of gemm.cu
int32_t dgc_gemm_nt(dgc_ctx *ctx, const float *a, const float *b, int M, int N, int K, float *c);
// the done counter of a reduction on the current stream
unsigned int *dgc_ctx_ticket(dgc_ctx *ctx);
// whether dgc_linear_bwd has a use for a transposed copy of the layer's input
bool dgc_linear_bwd_reads_t(int64_t M, int64_t K, int64_t N);
// dgc_linear_bwd, its weight gradients on the side stream where that helps (gemm.cu)
int32_t dgc_linear_bwd_beside(dgc_ctx *ctx, const float *a_dev, const float *w_dev, const float *c_dev, const float *dc_dev,
                              int32_t M, int32_t K, int32_t N, int32_t act, float *dz_dev, float *da_dev, float *dw_dev,
                              float *dbias_dev, const float *at_dev, bool *beside);
// true when dgc_gemm_nt() runs this shape on its persistent short-reduction tensor-core kernel
bool dgc_gemm_nt_persistent(const dgc_ctx *ctx, const float *a, int M, int N, int K);
const float2 *dgc_ctx_twiddles(dgc_ctx *ctx, int N);
// dgc_harmonic_render; by_partial: in FUNDAMENTAL mode one sine per partial and frame instead of groups of eight (osc_bank.cu)
int32_t dgc_harmonic_render_impl(dgc_ctx *ctx, const dgc_harmonic_params *p, const float *f0_dev, const float *uv_dev,
                                 const float *amps_dev, const float *gain_dev, float *scratch_dev, float *audio_dev,
                                 bool by_partial);
// dgc_onepole_fwd as three launches (linrec.cu)
int32_t dgc_onepole_in_passes(dgc_ctx *ctx, const float *x_dev, int32_t B, int32_t T, float a, float *y_dev);
// dgc_mss_loss_fwd with the voices in groups, each after its own event (mss_loss.cu)
constexpr int DGC_MSS_MAX_GROUPS = 4;
static inline int dgc_mss_group_start(int B, int q, int groups) { return (int)((int64_t)B * q / groups); }
int32_t dgc_mss_loss_fwd_groups(dgc_ctx *ctx, const dgc_mss_params *p, const float *pred_dev, const float *target_dev, int groups,
                                const cudaEvent_t *ready, double *loss_dev);

#define DGC_CUDA(ctx, call)                                                                  \
  do {                                                                                       \
    cudaError_t e__ = (call);                                                                \
    if (e__ != cudaSuccess)                                                                  \
      return dgc_fail(ctx, e__ == cudaErrorMemoryAllocation ? DGC_ERR_OOM : DGC_ERR_CUDA,    \
                      "%s: %s", #call, cudaGetErrorString(e__));                             \
  } while (0)

#define DGC_REQUIRE(ctx, cond, msg)                            \
  do {                                                         \
    if (!(cond)) return dgc_fail(ctx, DGC_ERR_INVALID, "%s: %s", __func__, msg); \
  } while (0)

#define DGC_LAUNCHED(ctx, name)                     \
  do {                                              \
    (ctx)->launches++;                              \
    int32_t rc__ = dgc_check_launch(ctx, name);     \
    if (rc__ != DGC_OK) return rc__;                \
  } while (0)

// ---- launches -----------------------------------------------------------------------------------------------------------
// Kernels of one stream follow each other by programmatic dependent launch: a kernel is set up on the SMs as soon as the last
// block of the kernel before has ended, and waits in dgc_after_previous() until that kernel's writes are visible.  Every kernel
// of the library calls it first thing, in every thread, before any early return: a grid that ended without having waited would
// let the one after it go on before the one in front of it was done.  After a copy, a memset or an event a launch waits as it
// always did.  A chain of short kernels is bound by what lies between them: 57 launches of a small training step took 421 us and
// take 303, eight of a small synthesis step 33 and 25.  Asking for the next kernel earlier, before the work
// (griddepcontrol.launch_dependents), sets its waiting blocks down beside the last ones of this kernel and beside the other
// stream's: 318 us for the same small training step, 2403 against 2349 for a large one.
__device__ __forceinline__ void dgc_after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A failed launch stays in cudaGetLastError (DGC_LAUNCHED reads it).
template <typename... P, typename... A>
static inline void dgc_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A &&...args) {
  cudaLaunchAttribute after;
  after.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  after.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &after;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

static inline int dgc_div_up(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }
static inline bool dgc_is_pow2(int n) { return n > 0 && (n & (n - 1)) == 0; }
