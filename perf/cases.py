"""The work that programs built on this framework have it do, as cases that can be timed.

Nine kinds of program, each through the Python binding of the C ABI:

  osc        oscillator bank -> one-pole filter -> magnitude spectra of the hops
  synth      harmonic+noise synthesis of a batch of voices and its multi-scale spectral loss, tensors on the GPU
  host       the same from and to page-locked host buffers, one blocking call per batch
  train      a whole training step of the controller, the synthesiser and the reverb
  biquad     tensor biquad bank, forward and reverse-time gradients
  reverb     partitioned convolution with a long impulse response, forward or forward and backward
  vocoder    buffer -> FFT -> phase vocoder -> inverse FFT -> overlap-add
  strip      one-pole -> compressor on every voice, modulated delay lines -> sample and hold on tensor lanes

Inputs are synthetic, drawn on the GPU from the seed; sizes follow the benchmark's configurations and the tests.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "dgen-audio_b200"))   # the working folder is the repository's root

import dgen_b200  # noqa: E402
from dgen_b200 import trainer, workloads  # noqa: E402

SIZES = (2048, 1024, 512, 256, 128, 64)   # windows of the spectral loss
SR = 16000.0


def listed():
    return [
        # One note of 64 partials through a filter and an analyser: the interactive size, a handful of small launches.
        dict(name="osc_64x65536", kind="osc", K=64, T=65536, N=1024, hop=256),
        # Half a second of two voices whose lengths fit no tile: one gradient-free evaluation while a user edits a patch.
        dict(name="synth_2x8191_ragged", kind="synth", B=2, T=8191, K=60, F=127, nbands=33, taps=129, replay=False),
        # The headline configuration: 16 voices of 4 s, the recorded step replayed as in a long run.
        dict(name="synth_16x64000_replay", kind="synth", B=16, T=64000, K=100, F=1000, nbands=65, taps=257, replay=True),
        # The throughput target: a whole dataset batch of 256 voices on one GPU, one call per batch.
        dict(name="synth_256x64000", kind="synth", B=256, T=64000, K=100, F=1000, nbands=65, taps=257, replay=False),
        # A host without tensors of its own (the C caller): everything goes up, loss and audio come back, every batch.
        dict(name="host_16x64000", kind="host", B=16, T=64000, K=100, F=1000, nbands=65, taps=257),
        # Fitting one short recording: few voices, a small controller, steps called one by one with a new batch each.
        dict(name="train_3x16001", kind="train", B=3, T=16001, K=60, F=250, nbands=65, taps=257, hidden=128,
             ir_len=4000, replay=False),
        # The training configuration: 32 voices per GPU, hidden 512, 1 s learnable impulse response, replayed.
        dict(name="train_32x64000_replay", kind="train", B=32, T=64000, K=100, F=1000, nbands=65, taps=257, hidden=512,
             ir_len=16000, replay=True),
        # A bank in a stream: state carried in and out, lanes and frames that fit no vector or chunk, any upstream
        # gradient, gradient of the input too.
        dict(name="biquad_5x37x50001_state", kind="biquad", B=5, L=37, T=50001, mode=1.0, loss="upstream"),
        # The bank at its full size: forward and BPTT of 256 lanes x 32 voices against a target.
        dict(name="biquad_32x256x262144", kind="biquad", B=32, L=256, T=262144, mode=0.0, loss="mse"),
        # Convolution reverb of 8 stereo pairs, 10 s at 48 kHz, 2 s impulse response.
        dict(name="reverb_16x480000", kind="reverb", V=16, T=480000, ir_len=96000, N=2048, hop=1024, backward=False),
        # Pitch shift of 8 channels by a ratio that moves from hop to hop.
        dict(name="vocoder_8x240000", kind="vocoder", V=8, T=240000, N=2048, hop=512),
        # The dynamics and delay part of a mixing desk: 64 channels and 64 lanes.
        dict(name="strip_64x262144", kind="strip", B=64, T=262144, lanes=64, max_delay=4800),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["osc", "synth", "synth", "host", "train", "biquad", "biquad", "reverb", "vocoder", "strip"])
    if kind == "osc":
        N = rng.choice([256, 512, 1024, 2048])
        return dict(kind=kind, K=_log_int(rng, 8, 256), T=_log_int(rng, 4096, 262144), N=N, hop=N // rng.choice([2, 4]))
    if kind in ("synth", "host", "train"):
        T = _log_int(rng, 4096, 64000)
        c = dict(kind=kind, B=_log_int(rng, 1, 256 if kind == "synth" else 32), T=T, K=rng.randint(20, 100),
                 F=max(2, T // rng.choice([64, 80, 128])))
        c["nbands"], c["taps"] = rng.choice([(65, 257), (65, 257), (33, 129), (65, 255)])
        if kind == "train":
            c.update(hidden=rng.choice([128, 256, 512]), ir_len=_log_int(rng, 1000, 16000))
        if kind != "host":
            c["replay"] = rng.random() < 0.5
        return c
    if kind == "biquad":
        L, T = _log_int(rng, 4, 256), _log_int(rng, 2048, 262144)
        B = _log_int(rng, 1, 32)
        if rng.random() < 0.5:      # the sizes of whole vectors and chunks are as common as the odd ones
            L, T = max(4, L // 4 * 4), T // 512 * 512
        return dict(kind=kind, B=B, L=L, T=T, mode=float(rng.randint(0, 5)), loss=rng.choice(["mse", "upstream"]))
    if kind == "reverb":
        N = rng.choice([512, 1024, 2048, 2048])
        T = _log_int(rng, 16000, 480000)
        return dict(kind=kind, V=_log_int(rng, 1, 16), T=T, ir_len=min(_log_int(rng, 2000, 96000), 190 * N // 2), N=N,
                    hop=N // 2, backward=rng.random() < 0.5)
    if kind == "vocoder":
        N = rng.choice([512, 1024, 2048])
        return dict(kind=kind, V=_log_int(rng, 1, 16), T=_log_int(rng, 16000, 240000), N=N, hop=N // 4)
    return dict(kind=kind, B=_log_int(rng, 1, 64), T=_log_int(rng, 2048, 262144), lanes=_log_int(rng, 1, 64),
                max_delay=_log_int(rng, 64, 9600))


# ---- what a program has in hand before the call -----------------------------------------------------------------------
_kept = {}


def _ctx():
    """One context per process, as a program on one GPU keeps it."""
    if "ctx" not in _kept:
        _kept["ctx"] = dgen_b200.Context(0)
    return _kept["ctx"]


def _stream():
    """The stream that recorded steps run on (a recording needs one that is not the default stream)."""
    if "stream" not in _kept:
        _kept["stream"] = torch.cuda.Stream()
    return _kept["stream"]


def _tap_matrix(nbands, taps):
    if (nbands, taps) not in _kept:
        _kept[nbands, taps] = torch.from_numpy(workloads.band_to_tap_matrix(nbands, taps)).cuda()
    return _kept[nbands, taps]


class _Draws:
    """Tensors drawn on the GPU from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def uniform(self, lo, hi, *shape):
        return torch.rand(*shape, generator=self.g, device="cuda") * (hi - lo) + lo

    def normal(self, sigma, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda") * sigma

    def log_uniform(self, lo, hi, *shape):
        return torch.exp(self.uniform(math.log(lo), math.log(hi), *shape))

    def curves(self, lo, hi, frames, *shape, span=40):
        """Control curves along the first axis: straight lines between random knots `span` frames apart."""
        knots = self.uniform(lo, hi, frames // span + 2, *shape)
        x = torch.arange(frames, device="cuda", dtype=torch.float32) / span
        i = x.floor().long()
        f = (x - i).reshape(-1, *([1] * len(shape)))
        return (knots[i] * (1 - f) + knots[i + 1] * f).contiguous()

    def tones(self, voices, frames, sr, lo=55.0, hi=880.0, partials=6, noise=0.02):
        """Recordings of steady notes with some noise: `partials` decaying harmonics per voice."""
        w = (2 * math.pi / sr) * self.log_uniform(lo, hi, voices, 1)
        n = torch.arange(frames, device="cuda", dtype=torch.float32)
        x = self.normal(noise, voices, frames)
        for k in range(1, partials + 1):
            x += torch.sin(torch.remainder(k * w * n, 2 * math.pi) + self.uniform(0, 6.28, voices, 1)) * (0.3 / k)
        return x


def _synth_inputs(c, seed):
    """Controls of the harmonic+noise synthesiser (f0: a random walk of half a semitone per control frame from
    55..880 Hz; amplitudes: slowly moving softmax; loudness and bands: curves in [0, 1]) and the recordings to match."""
    d, F, B, K, T = _Draws(seed), c["F"], c["B"], c["K"], c["T"]
    walk = torch.cumsum(d.normal(0.5, F, B), 0)
    f0 = (d.log_uniform(55.0, 880.0, B) * torch.exp2((walk - walk[:1]) / 12.0)).contiguous()
    amps = torch.softmax(d.normal(1.0, 1, B, K) + d.curves(-0.3, 0.3, F, B, K), dim=2)
    return dict(f0=f0, uv=torch.ones(F, B, device="cuda"), amps=amps, gain=d.curves(0.0, 1.0, F, B),
                noise_gain=d.curves(0.0, 1.0, F, B), bands=d.curves(0.0, 1.0, F, B, c["nbands"]),
                w=_tap_matrix(c["nbands"], c["taps"]), noise=d.normal(0.1, B, T), target=d.tones(B, T, SR))


def _synth_step(c):
    st = dgen_b200.HnStep()
    st.harm = dgen_b200.HarmonicParams(c["B"], c["T"], c["K"], c["F"], SR, 1.0, dgen_b200.PHASE_FUNDAMENTAL, 0)
    st.fir = dgen_b200.FirParams(c["B"], c["T"], c["F"], c["taps"], 0.12, 1)
    st.mss = dgen_b200.mss_params(c["B"], c["T"], SIZES)
    st.nbands = c["nbands"]
    return st


_ORDER = ("f0", "uv", "amps", "gain", "noise_gain", "bands", "w", "noise", "target")


def _synth_call(s):
    return s["ctx"].hn_forward_loss(s["step"], *s["inputs"], work=s["work"], loss=s["loss"], audio=s["audio"])


def _prepare_synth(c, seed):
    ctx, x = _ctx(), _synth_inputs(c, seed)
    s = dict(ctx=ctx, step=_synth_step(c), inputs=[x[k] for k in _ORDER], audio=torch.empty(c["B"], c["T"], device="cuda"),
             loss=torch.zeros(1, dtype=torch.float64, device="cuda"))
    n = int(ctx.lib.dgc_hn_forward_loss_work_floats(C.byref(s["step"])))
    s["work"] = torch.empty(n, device="cuda")
    if c["replay"]:
        st = s["stream"] = _stream()
        st.wait_stream(torch.cuda.current_stream())
        with ctx.on_stream(st), torch.cuda.stream(st):
            _synth_call(s)
            with ctx.record() as rec:
                _synth_call(s)
        s["graph"] = _Graphs([rec.graph])
    return s


class _Graphs:
    """Recordings that go with the state that owns them."""

    def __init__(self, graphs):
        self.graphs = graphs

    def __del__(self):
        for g in self.graphs:
            g.close()


def _run_synth(s):
    if "graph" not in s:
        _synth_call(s)
    else:
        cur, st = torch.cuda.current_stream(), s["stream"]
        st.wait_stream(cur)
        with s["ctx"].on_stream(st):
            s["graph"].graphs[0].launch()
        cur.wait_stream(st)
    return s["loss"], s["audio"]


def _prepare_host(c, seed):
    x = _synth_inputs(c, seed)
    return dict(ctx=_ctx(), step=_synth_step(c), inputs=[x[k].cpu().pin_memory() for k in _ORDER],
                audio=torch.empty(c["B"], c["T"]).pin_memory())


def _run_host(s):
    return s["ctx"].hn_forward_loss_host(s["step"], *s["inputs"], audio_out=s["audio"]), s["audio"]


class _Training:
    """A model with its batch.  Replayed: the batch lies in the model's own input buffers, as a loop that refills them
    in place keeps it.  Otherwise the batch comes as tensors of the caller's."""

    def __init__(self, c, seed):
        ctx, x = _ctx(), _synth_inputs(c, seed)
        B, F = c["B"], c["F"]
        self.model = m = trainer.HarmonicModel(
            ctx, B, c["T"], K=c["K"], F=F, sr=SR, nbands=c["nbands"], taps=c["taps"], hidden=c["hidden"],
            ir_len=c["ir_len"], sizes=SIZES, seed=int(seed), phase_mode=dgen_b200.PHASE_FUNDAMENTAL, counted_adam=True)
        pitch = (torch.log(x["f0"].clamp(min=1.0)) - math.log(40.0)) / math.log(2000.0 / 40.0)
        rows = torch.stack([pitch.reshape(-1), x["gain"].reshape(-1)], dim=1).contiguous()
        self.batch = [rows, x["f0"], x["uv"], x["gain"], x["noise_gain"], x["noise"], x["w"], x["target"]]
        m.step(*self.batch)
        if c["replay"]:
            self.batch = m.input_views()
            m.capture(*self.batch)

    def __del__(self):
        self.model.close()


def _prepare_train(c, seed):
    t = _Training(c, seed)
    return dict(training=t, replay=c["replay"])


def _run_train(s):
    m = s["training"].model
    loss = m.replay() if s["replay"] else m.step(*s["training"].batch)
    return dict(loss=loss, audio=m.out, grads=m.grads, params=m.params, m=m.m, v=m.v)


def _prepare_osc(c, seed):
    d = _Draws(seed)
    k = torch.arange(1, c["K"] + 1, device="cuda", dtype=torch.float32)
    n = torch.arange(c["N"], device="cuda", dtype=torch.float32)
    return dict(ctx=_ctx(), c=c, freq=k * d.uniform(55.0, 220.0, 1), amp=d.uniform(0.5, 1.0, c["K"]) / k,
                window=0.5 - 0.5 * torch.cos(n * (2 * math.pi / c["N"])))


def _run_osc(s):
    ctx, c = s["ctx"], s["c"]
    audio = ctx.osc_bank_const(s["freq"], s["amp"], c["T"], 44100.0)
    y = ctx.onepole_fwd(audio.view(1, -1), 0.9)
    return y, ctx.stft_mag(y, c["N"], c["hop"], s["window"])


def _prepare_biquad(c, seed):
    d, B, L, T = _Draws(seed), c["B"], c["L"], c["T"]
    s = dict(ctx=_ctx(), c=c, x=d.normal(1.0, B, T), cutoff=d.log_uniform(50.0, 8000.0, L), q=d.log_uniform(0.5, 8.0, L))
    if c["loss"] == "mse":
        s["target"] = d.normal(0.3, B, T, L)
    else:
        s["gy"] = d.normal(1e-3, B, T, L)
        s["state"] = torch.zeros(B, 4, L, device="cuda")
    return s


def _run_biquad(s):
    ctx, c = s["ctx"], s["c"]
    if c["loss"] == "mse":
        y = ctx.biquad_fwd(s["x"], s["cutoff"], s["q"], mode=c["mode"])
        return (y,) + ctx.biquad_mse_bwd(s["x"], s["cutoff"], s["q"], y, s["target"], loss_scale=1.0 / y.numel(),
                                         mode=c["mode"])
    y = ctx.biquad_fwd(s["x"], s["cutoff"], s["q"], mode=c["mode"], state=s["state"])
    return (y, s["state"]) + ctx.biquad_bwd(s["x"], s["cutoff"], s["q"], y, s["gy"], mode=c["mode"])


def _prepare_reverb(c, seed):
    d, n = _Draws(seed), c["ir_len"]
    fade = torch.exp(torch.arange(n, device="cuda", dtype=torch.float32) * (-6.91 / (0.6 * n)))
    s = dict(ctx=_ctx(), c=c, x=d.tones(c["V"], c["T"], 48000.0, noise=0.2), ir=d.normal(0.05, n) * fade)
    if c["backward"]:
        s["g"] = d.normal(1e-3, c["V"], c["T"])
    return s


def _run_reverb(s):
    ctx, c = s["ctx"], s["c"]
    y = ctx.partconv(s["x"], s["ir"], c["N"], c["hop"])
    if not c["backward"]:
        return y
    return (y,) + ctx.partconv_bwd(s["x"], s["ir"], c["N"], c["hop"], s["g"])


def _prepare_vocoder(c, seed):
    d, H = _Draws(seed), -(-c["T"] // c["hop"])
    n = torch.arange(c["N"], device="cuda", dtype=torch.float32)
    return dict(ctx=_ctx(), c=c, x=d.tones(c["V"], c["T"], 48000.0, noise=1e-3), ratio=d.curves(0.7, 1.4, H),
                window=0.5 - 0.5 * torch.cos(n * (2 * math.pi / c["N"])))


def _run_vocoder(s):
    ctx, c = s["ctx"], s["c"]
    re, im = ctx.stft(s["x"], c["N"], c["hop"], s["window"])
    re, im = ctx.phase_vocoder(re, im, s["ratio"], c["hop"])
    return ctx.istft_ola(re, im, c["T"], c["hop"], s["window"], gain=2.0 / 3.0)


def _prepare_strip(c, seed):
    d, B, T, W = _Draws(seed), c["B"], c["T"], c["lanes"]
    level = d.curves(0.05, 1.0, T, span=4000)
    return dict(ctx=_ctx(), x=d.tones(B, T, 48000.0, noise=0.05) * level, lanes=d.normal(0.3, T, W), c=c,
                delay=d.curves(0.0, c["max_delay"] - 1.0, T, span=2000), gate=(d.uniform(0, 1, T) > 0.97).float(),
                ring=torch.zeros(W, c["max_delay"], device="cuda"), head=torch.zeros(1, device="cuda"),
                held=torch.zeros(W, device="cuda"), y1=torch.zeros(B, device="cuda"), gr=torch.zeros(B, device="cuda"))


def _run_strip(s):
    ctx = s["ctx"]
    y = ctx.onepole_fwd(s["x"], 0.7, state=s["y1"])
    z = ctx.compressor(y, 4.0, -20.0, 6.0, 0.005, 0.05, 48000.0, state=s["gr"])
    d = ctx.delay_line(s["lanes"], s["delay"], s["c"]["max_delay"], ring=s["ring"], head=s["head"])
    h = ctx.latch(d, s["gate"], state=s["held"])
    return y, z, d, h, s["y1"], s["gr"], s["ring"], s["head"], s["held"]


_KINDS = {"osc": (_prepare_osc, _run_osc), "synth": (_prepare_synth, _run_synth), "host": (_prepare_host, _run_host),
          "train": (_prepare_train, _run_train), "biquad": (_prepare_biquad, _run_biquad),
          "reverb": (_prepare_reverb, _run_reverb), "vocoder": (_prepare_vocoder, _run_vocoder),
          "strip": (_prepare_strip, _run_strip)}


def prepare(case, seed):
    s = _KINDS[case["kind"]][0](case, seed)
    s["kind"] = case["kind"]
    return s


def run(state):
    return _KINDS[state["kind"]][1](state)


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def _fft(n):
    return 2.5 * n * math.log2(n)     # a real transform of n points


def _work(c):
    """(floats that have to be read or written once, operations)"""
    k = c["kind"]
    if k == "osc":
        H = -(-c["T"] // c["hop"])
        return 2 * c["K"] + c["T"] + H * (c["N"] // 2 + 1), 4.0 * c["K"] * c["T"] + H * _fft(c["N"])
    if k in ("synth", "host", "train"):
        B, T, K, F, nb, taps = c["B"], c["T"], c["K"], c["F"], c["nbands"], c["taps"]
        windows = sum(-(-T // (n // 4)) * B * 2 * _fft(n) for n in SIZES if n <= T)
        render = 2.0 * B * T * K + 4.0 * B * T * taps + 2.0 * F * B * nb * taps
        if k != "train":
            return F * B * (4 + K + nb) + taps * nb + 3 * B * T, render + windows
        h, rows, ir = c["hidden"], F * B, c["ir_len"]
        weights = 2 * h + 2 * h * h + h * (K + nb)
        params = weights + 3 * h + K + nb + ir
        H = -(-T // 1024) * B
        reverb = H * 2 * _fft(2048) + 8.0 * H * 1025 * -(-ir // 1024)
        # the backward repeats the products of the forward twice (inputs and weights) and its transforms once
        return (rows * 6 + taps * nb + 3 * B * T + 7 * params,
                2 * render + 2 * windows + 3 * reverb + 6.0 * rows * weights + 10.0 * params)
    if k == "biquad":
        n = c["B"] * c["T"] * c["L"]
        more = c["B"] * c["T"] if c["loss"] == "upstream" else 0
        return c["B"] * c["T"] + more + 3 * n + 4 * c["L"], 30.0 * n + (3.0 * n if more else 0.0)
    if k == "reverb":
        V, T, N = c["V"], c["T"], c["N"]
        H, P, nb = -(-T // c["hop"]) * V, -(-c["ir_len"] // c["hop"]), N // 2 + 1
        floats, ops = 2 * V * T + c["ir_len"], H * 2 * _fft(N) + P * _fft(N) + 8.0 * H * P * nb
        return (2 * floats, 3 * ops) if c["backward"] else (floats, ops)
    if k == "vocoder":
        H = -(-c["T"] // c["hop"]) * c["V"]
        return 2 * c["V"] * c["T"] + H, H * (2 * _fft(c["N"]) + 60.0 * c["N"])
    n, w = c["B"] * c["T"], c["T"] * c["lanes"]
    return 3 * n + 3 * w + 2 * c["T"] + c["lanes"] * (2 * c["max_delay"] + 2), 60.0 * n + 6.0 * w


def work(case):
    floats, ops = _work(case)
    return {"bytes": 4.0 * floats, "flops": float(ops)}


def tolerance(case):
    k = case["kind"]
    if k == "train":
        # the loss holds |a - b| of magnitudes: its gradient changes sign where they are equal within rounding, and
        # the step of an Adam update is of one size however small the gradient
        return {"rel": 1e-2, "max": 0.5}
    if k == "biquad":
        return {"rel": 1e-3, "max": 3e-2}     # poles at 0.9994: 32-bit sums of the recurrence differ by 2e-4 of the peak
    if k == "vocoder":
        # phases of bins with hardly any energy are decided by rounding, and errors of a phase add up over the hops
        return {"rel": 1e-2, "max": 0.5}
    if k in ("synth", "host"):
        return {"rel": 1e-4, "max": 2e-3}     # phases of up to 100 f0 in 32 bits, single-precision sines
    return {"rel": 2e-5, "max": 1e-3}
