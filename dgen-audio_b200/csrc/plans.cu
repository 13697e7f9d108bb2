// Composite entry points that take HOST buffers: what a host calls once per batch.  They own a
// device staging area inside the context, enqueue one asynchronous copy per input straight from the
// caller's buffers (full PCIe rate when those are page-locked) on an upload stream, in the order the
// kernels need them, and the kernels on the context stream behind per-group events: the render starts
// as soon as its control tables have landed, while the noise inputs and the target are still in
// flight.  The result returns to host memory.
#include "common.cuh"
#include <cstdlib>
#include <cstring>

namespace {

// device staging area carved into sub-buffers, grown on demand
struct Carver {
  float *base;
  uint64_t used = 0;
  explicit Carver(float *b) : base(b) {}
  float *take(uint64_t n) {
    float *p = base + used;
    used += (n + 63) & ~63ull;  // keep every sub-buffer 256-byte aligned
    return p;
  }
};

int32_t ensure_stage(dgc_ctx *ctx, uint64_t nfloats) {
  if (nfloats <= ctx->stage_floats) return DGC_OK;
  if (ctx->stage_dev) {
    cudaStreamSynchronize(ctx->stream);
    cudaFree(ctx->stage_dev);
    ctx->buffer_generation++;
    ctx->stage_dev = nullptr;
    ctx->stage_floats = 0;
  }
  DGC_CUDA(ctx, cudaMalloc(&ctx->stage_dev, nfloats * sizeof(float)));
  ctx->stage_floats = nfloats;
  return DGC_OK;
}

// out may be the same buffer as a (element i is read before it is written): no restrict on those two
__global__ void add2_kernel(const float *a, const float *__restrict__ b, size_t n, float *out) {
  dgc_after_previous();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = __fadd_rn(a[i], b[i]);
}

}  // namespace

DGC_EXPORT uint64_t dgc_hn_forward_loss_work_floats(const dgc_hn_step *s) {
  if (!s || s->harm.B <= 0 || s->harm.T <= 0 || s->harm.F <= 0) return 0;
  const uint64_t nBT = ((uint64_t)s->harm.B * s->harm.T + 63) & ~63ull;
  const uint64_t taps = (s->fir.taps > 0 && s->nbands > 0) ? (((uint64_t)s->harm.F * s->harm.B * s->fir.taps + 63) & ~63ull) : 0;
  return 2 * nBT + taps + 64;
}

// Device-resident forward + loss.  The harmonic branch (track, chunk sums, scan, render) and the noise branch
// (band -> tap map, FIR) share no data until the loss, so they run on two streams: the small or latency-bound
// kernels of one chain (the 64-block phase scan, the band -> tap matmul) and the last waves of the big ones fill
// under the other chain's work.  The loss reads the prediction as the sum of the two branch outputs.
// The host-buffer variant uploads on its own stream while the first kernels already run, and reads the audio back while the
// loss is still being computed:
struct HostEvents {
  cudaEvent_t noise_inputs;       // the noise branch's inputs are in device memory
  const cudaEvent_t *target;      // group q of the target's voices is
  int groups;
  cudaEvent_t audio;              // recorded when the audio is complete
};
static int32_t hn_forward_loss_impl(dgc_ctx *ctx, const dgc_hn_step *s, const float *f0_dev, const float *uv_dev,
                                    const float *amps_dev, const float *gain_dev, const float *noise_gain_dev,
                                    const float *taps_or_bands_dev, const float *w_dev, const float *noise_dev,
                                    const float *target_dev, float *work_dev, double *loss_dev, float *audio_dev,
                                    const HostEvents *ev) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, s && f0_dev && uv_dev && amps_dev && gain_dev && target_dev && loss_dev && work_dev, "null pointer");
  const int B = s->harm.B, T = s->harm.T, K = s->harm.K, F = s->harm.F;
  DGC_REQUIRE(ctx, B > 0 && T > 0 && K > 0 && F > 0, "size out of range");
  const int NT = s->fir.taps, NB = s->nbands;
  const bool noise = NT > 0;
  if (noise) {
    DGC_REQUIRE(ctx, noise_gain_dev && taps_or_bands_dev && noise_dev, "noise branch needs its inputs");
    DGC_REQUIRE(ctx, s->fir.B == B && s->fir.T == T && s->fir.F == F, "fir shape differs from harmonic shape");
    DGC_REQUIRE(ctx, NB == 0 || w_dev, "band synthesis needs the matrix W");
  }
  DGC_REQUIRE(ctx, s->mss.B == B && s->mss.T == T, "loss shape differs from harmonic shape");
  DGC_REQUIRE(ctx, (((uintptr_t)work_dev) & 15) == 0, "work buffer must be 16-byte aligned");
  const uint64_t nBT = (uint64_t)B * T, nFB = (uint64_t)F * B;
  Carver wc(work_dev);
  float *d_harm = wc.take(nBT), *d_noise = noise ? wc.take(nBT) : nullptr;
  float *d_taps = (noise && NB > 0) ? wc.take(nFB * NT) : const_cast<float *>(taps_or_bands_dev);
  // Size the context scratch for the largest user BEFORE the streams fork: growing it later would free a buffer
  // the other stream may still be reading.
  {
    uint64_t need = dgc_harmonic_scratch_floats(&s->harm), m = dgc_mss_partial_floats(&s->mss) + 4;
    if (m > need) need = m;
    if (!dgc_ctx_scratch(ctx, need)) return DGC_ERR_OOM;
  }
  if (!ctx->aux_stream) {
    DGC_CUDA(ctx, cudaStreamCreateWithFlags(&ctx->aux_stream, cudaStreamNonBlocking));
    DGC_CUDA(ctx, cudaEventCreateWithFlags(&ctx->fork_ev, cudaEventDisableTiming));
    DGC_CUDA(ctx, cudaEventCreateWithFlags(&ctx->join_ev, cudaEventDisableTiming));
  }
  // tables cached per (F, T) are built on first use by a kernel on the current stream: make sure they exist
  // before the streams fork, so that neither branch picks up a table the other one is still writing
  if (!dgc_ctx_row_table(ctx, F, T)) return DGC_ERR_CUDA;
  int32_t rc = DGC_OK;
  cudaStream_t main_stream = ctx->stream;
  bool forked = false;
  // From a few million samples per step on, every big kernel fills the GPU by itself and running the FIR beside the
  // render buys nothing: then only the band -> tap map runs on the side stream, and the FIR follows the render on
  // the caller's stream ADDING into the render's output, which drops the pass that sums the two branches (the sum
  // is the same single-precision add either way: the results are bit-identical).  DGC_HN_FIR=side|serial forces one.
  static const int fir_mode = [] {
    const char *e = getenv("DGC_HN_FIR");
    return !e ? 0 : strcmp(e, "side") == 0 ? 1 : strcmp(e, "serial") == 0 ? 2 : 0;
  }();
  const bool serial_fir = noise && (fir_mode == 2 || (fir_mode == 0 && nBT >= (4ull << 20)));
  // nothing is added later: the branch (and the FIR behind it) writes where the caller wants the audio, unless an input that is
  // still to be read lies there
  auto holds = [&](const float *p, uint64_t n) { return p && p < audio_dev + nBT && audio_dev < p + n; };
  const bool holds_input = holds(f0_dev, nFB) || holds(uv_dev, nFB) || holds(amps_dev, nFB * K) || holds(gain_dev, nFB) ||
                           (noise && (holds(noise_gain_dev, nFB) || holds(taps_or_bands_dev, nFB * (NB > 0 ? NB : NT)) ||
                                      holds(NB > 0 ? w_dev : nullptr, (uint64_t)NT * NB) || holds(noise_dev, nBT)));
  if (audio_dev && (serial_fir || !noise) && (((uintptr_t)audio_dev) & 15) == 0 && !holds_input) d_harm = audio_dev;
  if (noise) {
    // fork: the noise branch starts where the caller's stream stands now
    DGC_CUDA(ctx, cudaEventRecord(ctx->fork_ev, main_stream));
    DGC_CUDA(ctx, cudaStreamWaitEvent(ctx->aux_stream, ctx->fork_ev, 0));
    if (ev) DGC_CUDA(ctx, cudaStreamWaitEvent(ctx->aux_stream, ev->noise_inputs, 0));
    forked = true;
    ctx->stream = ctx->aux_stream;
    if (NB > 0) rc = dgc_bands_to_taps(ctx, taps_or_bands_dev, w_dev, (int32_t)nFB, NB, NT, d_taps);
    if (rc == DGC_OK && !serial_fir) {
      dgc_fir_params fp = s->fir;
      fp.accumulate = 0;
      rc = dgc_fir_noise(ctx, &fp, noise_dev, d_taps, noise_gain_dev, d_noise);
    }
    cudaError_t e = cudaEventRecord(ctx->join_ev, ctx->aux_stream);
    ctx->stream = main_stream;
    if (rc == DGC_OK && e != cudaSuccess) rc = dgc_fail(ctx, DGC_ERR_CUDA, "event record: %s", cudaGetErrorString(e));
  }
  // the harmonic branch goes onto the caller's stream BEFORE that stream is told to wait for the noise branch
  if (rc == DGC_OK) {
    dgc_harmonic_params hp = s->harm;
    hp.accumulate = 0;
    rc = dgc_harmonic_render(ctx, &hp, f0_dev, uv_dev, amps_dev, gain_dev, nullptr, d_harm);
  }
  // join, whatever happened above: nothing of this call is left running beside the caller's stream
  if (forked) cudaStreamWaitEvent(main_stream, ctx->join_ev, 0);
  if (rc != DGC_OK) return rc;
  if (serial_fir) {
    dgc_fir_params fp = s->fir;
    fp.accumulate = 1;
    rc = dgc_fir_noise(ctx, &fp, noise_dev, d_taps, noise_gain_dev, d_harm);
    if (rc != DGC_OK) return rc;
  }
  // the sum of the branches: in the audio buffer when the caller wants it, else in place (measured 0.349 ms per step
  // against 0.360 ms with the loss kernel adding the two signals as it loads them)
  float *mix = audio_dev ? audio_dev : d_harm;
  if (noise && !serial_fir) {
    dgc_launch(add2_kernel, dgc_div_up((int64_t)nBT, 256), 256, 0, ctx->stream, d_harm, d_noise, nBT, mix);
    DGC_LAUNCHED(ctx, "add_branches");
  } else if (mix != d_harm) {
    DGC_CUDA(ctx, cudaMemcpyAsync(mix, d_harm, nBT * sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
  }
  if (ev) {
    DGC_CUDA(ctx, cudaEventRecord(ev->audio, main_stream));
    return dgc_mss_loss_fwd_groups(ctx, &s->mss, mix, target_dev, ev->groups, ev->target, loss_dev);
  }
  return dgc_mss_loss_fwd(ctx, &s->mss, mix, target_dev, nullptr, loss_dev);
}

DGC_EXPORT int32_t dgc_hn_forward_loss(dgc_ctx *ctx, const dgc_hn_step *s, const float *f0_dev, const float *uv_dev,
                                       const float *amps_dev, const float *gain_dev, const float *noise_gain_dev,
                                       const float *taps_or_bands_dev, const float *w_dev, const float *noise_dev,
                                       const float *target_dev, float *work_dev, double *loss_dev, float *audio_dev) {
  return hn_forward_loss_impl(ctx, s, f0_dev, uv_dev, amps_dev, gain_dev, noise_gain_dev, taps_or_bands_dev, w_dev,
                              noise_dev, target_dev, work_dev, loss_dev, audio_dev, nullptr);
}

// slot < 0: the blocking call (one staging area, returns after the loss has arrived).
// slot 0 / 1: one of two steps in flight -- inputs go to the slot's own staging area, so the upload of the next
// step crosses PCIe while this step computes; nothing is waited for here (dgc_hn_forward_loss_host_wait does).
static int32_t hn_host_enqueue(dgc_ctx *ctx, const dgc_hn_step *s, const float *f0_host, const float *uv_host,
                               const float *amps_host, const float *gain_host, const float *noise_gain_host,
                               const float *taps_or_bands_host, const float *w_host, const float *noise_host,
                               const float *target_host, double *loss_host, float *audio_host, int slot) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, s && f0_host && uv_host && amps_host && gain_host && loss_host, "null pointer");
  DGC_REQUIRE(ctx, target_host || s->target_dev, "the target must be given in host memory or as a resident device buffer");
  const int B = s->harm.B, T = s->harm.T, K = s->harm.K, F = s->harm.F;
  DGC_REQUIRE(ctx, B > 0 && T > 0 && K > 0 && F > 0, "size out of range");
  const int NT = s->fir.taps, NB = s->nbands;
  const bool noise = NT > 0;
  if (noise) {
    DGC_REQUIRE(ctx, noise_gain_host && taps_or_bands_host && (noise_host || s->noise_seed), "noise branch needs its inputs");
    DGC_REQUIRE(ctx, s->fir.B == B && s->fir.T == T && s->fir.F == F, "fir shape differs from harmonic shape");
    DGC_REQUIRE(ctx, NB == 0 || w_host, "band synthesis needs the matrix W");
  }
  DGC_REQUIRE(ctx, s->mss.B == B && s->mss.T == T, "loss shape differs from harmonic shape");
  const bool gen_noise = noise && !noise_host;          // generated on the device from s->noise_seed
  const bool resident_target = s->target_dev != nullptr;
  const uint64_t nFB = (uint64_t)F * B, nBT = (uint64_t)B * T;
  const uint64_t n_tab = noise ? nFB * (NB > 0 ? NB : NT) : 0;
  const uint64_t n_w = (noise && NB > 0) ? (uint64_t)NT * NB : 0;
  // host -> device inputs, in one contiguous pinned block
  const uint64_t in_floats = 3 * nFB + nFB * K + (noise ? nFB + n_tab + n_w + nBT : 0) + nBT;
  const uint64_t dev_extra = nBT /*audio*/ + dgc_hn_forward_loss_work_floats(s) + 64 * 16;
  const bool piped = slot >= 0;
  if (!piped)
    DGC_REQUIRE(ctx, !ctx->pipe_pending[0] && !ctx->pipe_pending[1],
                "steps submitted with dgc_hn_forward_loss_host_submit are still in flight: wait for them first");
  int32_t rc = ensure_stage(ctx, (piped ? 0 : in_floats) + dev_extra + 64 * 16);
  if (rc != DGC_OK) return rc;

  // each on its own: what a failed call left out, the next one makes
  auto need_stream = [](cudaStream_t &s) { return s ? cudaSuccess : cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking); };
  auto need_event = [](cudaEvent_t &e) { return e ? cudaSuccess : cudaEventCreateWithFlags(&e, cudaEventDisableTiming); };
  DGC_CUDA(ctx, need_stream(ctx->copy_stream));
  DGC_CUDA(ctx, need_stream(ctx->out_stream));
  for (auto &e : ctx->copy_ev) DGC_CUDA(ctx, need_event(e));
  DGC_CUDA(ctx, need_event(ctx->audio_ev));
  DGC_CUDA(ctx, need_event(ctx->out_ev));
  if (!ctx->status_host) DGC_CUDA(ctx, cudaMallocHost(&ctx->status_host, sizeof(int32_t)));
  cudaEvent_t *ev = ctx->copy_ev;
  if (piped) {
    const uint64_t need = in_floats + 64 * 16;
    if (ctx->pipe_in_floats[slot] < need) {
      if (ctx->pipe_in[slot]) {
        cudaStreamSynchronize(ctx->stream);
        cudaStreamSynchronize(ctx->copy_stream);
        cudaFree(ctx->pipe_in[slot]);
        ctx->buffer_generation++;
        ctx->pipe_in[slot] = nullptr;
        ctx->pipe_in_floats[slot] = 0;
      }
      DGC_CUDA(ctx, cudaMalloc(&ctx->pipe_in[slot], need * sizeof(float)));
      ctx->pipe_in_floats[slot] = need;
    }
    DGC_CUDA(ctx, need_event(ctx->pipe_done[slot]));
    for (auto &e : ctx->pipe_ev[slot]) DGC_CUDA(ctx, need_event(e));
    ev = ctx->pipe_ev[slot];
    // the slot's previous step may still read its staging area: the new upload waits for that step's end
    if (ctx->pipe_pending[slot])
      return dgc_fail(ctx, DGC_ERR_INVALID, "slot %d still holds a step: call dgc_hn_forward_loss_host_wait first", slot);
    if (ctx->pipe_used[slot]) DGC_CUDA(ctx, cudaStreamWaitEvent(ctx->copy_stream, ctx->pipe_done[slot], 0));
  }
  // Blocking form: every earlier call ended with a stream synchronisation, so no kernel still reads the staging
  // area; work the caller queued on the context stream before this call does not touch it either.
  Carver dc(piped ? ctx->pipe_in[slot] : ctx->stage_dev);
  cudaError_t cp_err = cudaSuccess;
  cudaStream_t up = ctx->copy_stream;
  auto put = [&](const float *src, uint64_t n) -> float * {
    float *d = dc.take(n);
    cudaError_t e = cudaMemcpyAsync(d, src, n * sizeof(float), cudaMemcpyHostToDevice, up);
    if (e != cudaSuccess && cp_err == cudaSuccess) cp_err = e;
    return d;
  };
  auto mark = [&](int i) {
    cudaError_t e = cudaEventRecord(ev[i], up);
    if (e != cudaSuccess && cp_err == cudaSuccess) cp_err = e;
  };
  // The small inputs cost 5 us and a gap each on the link whatever their size: up to 512 KB of them are gathered in
  // page-locked memory, while the amplitudes are already crossing, and go up as one copy.
  const uint64_t small_floats = (noise ? 4 : 3) * ((nFB + 63) & ~63ull) + ((n_w + 63) & ~63ull);
  float *gather = nullptr;
  if (small_floats <= (128u << 10)) {
    const int k = piped ? 1 + slot : 0;
    if (ctx->pinned_floats[k] < small_floats) {
      if (ctx->pinned[k]) cudaFreeHost(ctx->pinned[k]);
      ctx->pinned[k] = nullptr;
      ctx->pinned_floats[k] = 0;
      DGC_CUDA(ctx, cudaMallocHost(&ctx->pinned[k], small_floats * sizeof(float)));
      ctx->pinned_floats[k] = small_floats;
    }
    gather = ctx->pinned[k];
  }
  // group 0: harmonic controls; group 1: noise branch; then the target, in groups of voices so that the loss of the first
  // ones is computed while the last are on their way
  float *d_amps = put(amps_host, nFB * K);
  float *d_small = dc.take(small_floats), *d_next = d_small;
  auto put_small = [&](const float *src, uint64_t n) -> float * {
    float *d = d_next;
    d_next += (n + 63) & ~63ull;
    if (gather) memcpy(gather + (d - d_small), src, n * sizeof(float));
    else {
      cudaError_t e = cudaMemcpyAsync(d, src, n * sizeof(float), cudaMemcpyHostToDevice, up);
      if (e != cudaSuccess && cp_err == cudaSuccess) cp_err = e;
    }
    return d;
  };
  float *d_f0 = put_small(f0_host, nFB), *d_uv = put_small(uv_host, nFB), *d_gain = put_small(gain_host, nFB);
  float *d_ng = noise ? put_small(noise_gain_host, nFB) : nullptr, *d_w = n_w ? put_small(w_host, n_w) : nullptr;
  if (gather) {
    cudaError_t e = cudaMemcpyAsync(d_small, gather, small_floats * sizeof(float), cudaMemcpyHostToDevice, up);
    if (e != cudaSuccess && cp_err == cudaSuccess) cp_err = e;
  }
  mark(0);
  float *d_tab = nullptr, *d_noise = nullptr;
  if (noise) {
    d_tab = put(taps_or_bands_host, n_tab);
    d_noise = gen_noise ? dc.take(nBT) : put(noise_host, nBT);
  }
  mark(1);
  // four groups, each loss launch still a few waves of blocks; a resident target is one group that waits for nothing
  const int groups = !resident_target && B >= 8 && nBT >= (1u << 18) ? DGC_MSS_MAX_GROUPS : 1;
  float *d_target = resident_target ? const_cast<float *>(s->target_dev) : dc.take(nBT);
  for (int q = 0; q < groups; ++q) {
    const uint64_t t0 = (uint64_t)dgc_mss_group_start(B, q, groups) * T, t1 = (uint64_t)dgc_mss_group_start(B, q + 1, groups) * T;
    if (!resident_target) {
      cudaError_t e = cudaMemcpyAsync(d_target + t0, target_host + t0, (t1 - t0) * sizeof(float), cudaMemcpyHostToDevice, up);
      if (e != cudaSuccess && cp_err == cudaSuccess) cp_err = e;
    }
    mark(2 + q);
  }
  if (cp_err != cudaSuccess) {
    cudaStreamSynchronize(ctx->copy_stream);
    return dgc_fail(ctx, DGC_ERR_CUDA, "input upload: %s", cudaGetErrorString(cp_err));
  }
  // from here on every exit path drains the upload stream before returning (the caller may reuse or free
  // its buffers as soon as this function returns)
  auto bail = [&](int32_t code) {
    cudaStreamSynchronize(ctx->copy_stream);
    cudaStreamSynchronize(ctx->stream);
    cudaStreamSynchronize(ctx->out_stream);
    return code;
  };
  // device work area of the two-branch step, and (only when the caller wants the audio back) the summed signal
  dgc_hn_step st = *s;
  // (two steps in flight share ONE work area: their kernels run one after the other on the context stream)
  Carver wc(ctx->stage_dev);
  Carver &work_carver = piped ? wc : dc;
  float *d_work = work_carver.take(dgc_hn_forward_loss_work_floats(&st));
  float *d_audio = audio_host ? work_carver.take(nBT) : nullptr;
  // the harmonic branch only needs group 0; the noise branch and the loss wait for their own uploads inside
  if (cudaStreamWaitEvent(ctx->stream, ev[0], 0) != cudaSuccess) return bail(dgc_fail(ctx, DGC_ERR_CUDA, "event wait"));
  if (gen_noise) {   // on the context stream, before the step forks its noise branch off it
    rc = dgc_noise_fill(ctx, s->noise_seed, s->noise_mode, B, T, s->noise_sigma, d_noise);
    if (rc != DGC_OK) return bail(rc);
  }
  double *loss_dev = ctx->loss_accum + (piped ? 1 + slot : 0);
  const HostEvents events = {ev[1], ev + 2, groups, ctx->audio_ev};
  rc = hn_forward_loss_impl(ctx, &st, d_f0, d_uv, d_amps, d_gain, d_ng, d_tab, d_w, d_noise, d_target, d_work, loss_dev,
                            d_audio, &events);
  if (rc != DGC_OK) return bail(rc);
  cudaError_t e = cudaSuccess;
  auto next = [&](cudaError_t r) {   // the first error stands, what follows it is still enqueued
    if (e == cudaSuccess) e = r;
  };
  if (audio_host) {   // the way down is free while the target comes up and the loss is computed
    next(cudaStreamWaitEvent(ctx->out_stream, ctx->audio_ev, 0));
    if (e == cudaSuccess)
      next(cudaMemcpyAsync(audio_host, d_audio, nBT * sizeof(float), cudaMemcpyDeviceToHost, ctx->out_stream));
    next(cudaEventRecord(ctx->out_ev, ctx->out_stream));
  }
  next(cudaMemcpyAsync(loss_host, loss_dev, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  if (!piped) next(cudaMemcpyAsync(ctx->status_host, ctx->status_dev, sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
  // the step ends when its audio is down too: the next one writes the same buffer
  if (audio_host) next(cudaStreamWaitEvent(ctx->stream, ctx->out_ev, 0));
  if (piped) next(cudaEventRecord(ctx->pipe_done[slot], ctx->stream));
  if (!piped || e != cudaSuccess) next(cudaStreamSynchronize(ctx->stream));
  if (e != cudaSuccess) return bail(dgc_fail(ctx, DGC_ERR_CUDA, "end of the step: %s", cudaGetErrorString(e)));
  if (!piped) return dgc_report_status(ctx, *ctx->status_host);
  ctx->pipe_used[slot] = true;
  ctx->pipe_pending[slot] = true;
  return DGC_OK;
}

DGC_EXPORT int32_t dgc_hn_forward_loss_host(dgc_ctx *ctx, const dgc_hn_step *s, const float *f0_host,
                                            const float *uv_host, const float *amps_host, const float *gain_host,
                                            const float *noise_gain_host, const float *taps_or_bands_host,
                                            const float *w_host, const float *noise_host, const float *target_host,
                                            double *loss_host, float *audio_host) {
  return hn_host_enqueue(ctx, s, f0_host, uv_host, amps_host, gain_host, noise_gain_host, taps_or_bands_host, w_host,
                         noise_host, target_host, loss_host, audio_host, -1);
}

DGC_EXPORT int32_t dgc_hn_forward_loss_host_submit(dgc_ctx *ctx, const dgc_hn_step *s, const float *f0_host,
                                                   const float *uv_host, const float *amps_host,
                                                   const float *gain_host, const float *noise_gain_host,
                                                   const float *taps_or_bands_host, const float *w_host,
                                                   const float *noise_host, const float *target_host, int32_t slot,
                                                   double *loss_host, float *audio_host) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, slot == 0 || slot == 1, "slot must be 0 or 1");
  return hn_host_enqueue(ctx, s, f0_host, uv_host, amps_host, gain_host, noise_gain_host, taps_or_bands_host, w_host,
                         noise_host, target_host, loss_host, audio_host, slot);
}

DGC_EXPORT int32_t dgc_hn_forward_loss_host_wait(dgc_ctx *ctx, int32_t slot) {
  if (!ctx) return DGC_ERR_INVALID;
  DGC_REQUIRE(ctx, slot == 0 || slot == 1, "slot must be 0 or 1");
  DGC_REQUIRE(ctx, ctx->pipe_pending[slot], "no step was submitted on this slot");
  ctx->pipe_pending[slot] = false;
  DGC_CUDA(ctx, cudaEventSynchronize(ctx->pipe_done[slot]));
  return DGC_OK;
}
