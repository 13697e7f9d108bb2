"""The harmonic render in groups of eight partials, where its grouping can go wrong: fewer partials than a group, one more or
one less than whole groups, rows that no 16-byte load fits, counts that change inside a warp, phases at zero and half turns."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

import dgen_b200  # noqa: E402
from oracle import torch_oracle as to  # noqa: E402

SR = 16000.0


@pytest.fixture(scope="module")
def ctx():
    return dgen_b200.Context(0)


def _render(ctx, f0, amps, T, scratch=None):
    F, B, _ = amps.shape
    one = torch.ones(F, B, device="cuda")
    return ctx.harmonic_render(f0.cuda(), one, amps.cuda(), one, T, SR, phase_mode=dgen_b200.PHASE_FUNDAMENTAL, scratch=scratch)


def _double(f0, amps, T):
    """The same sums in double on the single-precision track, phases as exact multiples of its running sum."""
    F, B, K = amps.shape
    rows = to.rows_of(F, T)
    lo, hi, fr = (torch.as_tensor(np.asarray(r)) for r in rows)
    lo, hi, fr = lo.long(), hi.long(), fr.float()[:, None]
    f = (1 - fr) * f0[lo] + fr * f0[hi]
    inc = f.double() / SR
    ph = torch.remainder(torch.cumsum(inc, 0) - inc, 1.0)
    k = torch.arange(1, K + 1).float()
    a = ((1 - fr.double())[..., None] * amps[lo].double() + fr.double()[..., None] * amps[hi].double())
    a = a * (f[..., None] * k < SR / 2)
    s = (a * torch.sin(2 * np.pi * torch.remainder(ph[..., None] * k.double(), 1.0))).sum(2)
    return (s / (a.sum(2) + 1e-8)).T


@pytest.mark.parametrize("K", [1, 3, 7, 8, 9, 15, 16, 17, 36, 41, 100, 129])
@pytest.mark.parametrize("f_hi", [60.0, 900.0])
def test_groups_of_partials_against_double(ctx, K, f_hi):
    g = torch.Generator().manual_seed(K)
    B, F, T = 3, 9, 603
    f0 = torch.rand(F, B, generator=g) * (f_hi - 50.0) + 50.0       # up to 900 Hz: the audible count moves by several a warp
    amps = torch.rand(F, B, K, generator=g)
    got = _render(ctx, f0, amps, T).cpu().double()
    want = _double(f0, amps, T)
    # a mean of sines: each good to a few 2^-24, its phase to 2^-33 turns a frame of the track's rounded advance
    assert (got - want).abs().max() < 1e-6 + 2 * np.pi * K * T * 2.0 ** -33


def test_zero_and_quarter_turn_phases(ctx):
    """f0 = 0 keeps every phase at zero: sums of exact zeros.  f0 = sr / 4 walks quarter turns, where the angles change sides."""
    F, B, K, T = 4, 2, 24, 256
    f0 = torch.zeros(F, B)
    f0[:, 1] = SR / 4
    amps = torch.rand(F, B, K, generator=torch.Generator().manual_seed(1)) + 0.1
    amps[:, 1, 1:] = 0.0          # partial 2 is at Nyquist or, by the rounding of the track, just below
    got = _render(ctx, f0, amps, T).cpu().double()
    assert torch.equal(got[0], torch.zeros(T).double())
    want = torch.sin(torch.pi / 2 * torch.arange(T, dtype=torch.float64))
    # the interpolated f0 is a unit in the last place off in some frames: 2^-24 / 4 turns each
    assert (got[1] - want).abs().max() < 3e-7 + T * 2.0 ** -26 * 2 * np.pi


def test_the_last_row_is_not_read_past_its_end(ctx):
    """K of no whole group, every partial audible, NaN behind the last row: nothing of it comes in."""
    F, B, K, T = 5, 1, 12, 300
    f0 = torch.full((F, B), 100.0)
    room = torch.full((F * B * K + 8,), float("nan"), device="cuda")
    room[:F * B * K] = torch.rand(F * B * K, device="cuda")
    amps = room[:F * B * K].view(F, B, K)
    one = torch.ones(F, B, device="cuda")
    y = ctx.harmonic_render(f0.cuda(), one, amps, one, T, SR, phase_mode=dgen_b200.PHASE_FUNDAMENTAL)
    assert torch.isfinite(y).all()


def _exact_phases(K, counts, spectrum, B, T, seed):
    """One control row: a constant f0 whose increment is a whole number m of 2^-32 turns, so that every phase is known exactly.
    counts: audible partials, one voice each.  Returns f0, amplitudes and the sums in double."""
    rng = np.random.default_rng(seed)
    # count = the largest k with k m < 2^31; m of 24 bits at most (f0 and the increment are then exact in single precision)
    m = np.array([int((2 ** 31 - 1) // (c + 0.5)) for c in counts], dtype=np.int64)
    shift = np.maximum(0, np.ceil(np.log2(m)).astype(np.int64) - 24)
    m = (m >> shift) << shift
    assert all((2 ** 31 - 1) // v == c for v, c in zip(m.tolist(), counts))
    amps = rng.uniform(0.0, 1.0, (1, B, K)).astype(np.float32)
    if spectrum == "last":                      # all of it in the last eight audible partials
        for b, c in enumerate(counts):
            amps[0, b, :max(0, min(c, K) - 8)] = 0.0
    n = np.arange(T, dtype=np.uint64)
    want = np.zeros((B, T))
    for b, c in enumerate(counts):
        for k in range(1, min(c, K) + 1):
            turns = ((n * np.uint64(k * int(m[b]))) & np.uint64(2 ** 32 - 1)).astype(np.float64) * 2.0 ** -32
            want[b] += amps[0, b, k - 1].astype(np.float64) * np.sin(2 * np.pi * turns)
        want[b] /= amps[0, b, :min(c, K)].astype(np.float64).sum() + 1e-8
    sr = 65536.0
    return torch.from_numpy((m * 2.0 ** -32 * sr).astype(np.float32))[None], torch.from_numpy(amps), want, sr


def _norm_error(got, want):
    return float(np.linalg.norm(got - want) / np.linalg.norm(want))


# A sine partial by partial is off by 3.6e-7 (the fast sine) and 2^-24 turns (23 bits of phase), 5.5e-7 of its 0.71 when the two
# are spread evenly, whatever the count: a render in groups is not allowed to lose that, on any row or spectrum.
PER_PARTIAL = 6e-7


@pytest.mark.parametrize("spectrum", ["flat", "last"])
@pytest.mark.parametrize("K", [8, 63, 64, 65, 100, 104, 105, 128, 129, 257, 512])
def test_error_does_not_grow_with_the_partials(ctx, K, spectrum):
    """Rows at the edges of groups, of a polynomial's segment and of the rule by which rows are cut into segments; all partials of
    the row audible, or one group, one segment less."""
    counts = [K, max(1, K - 8), max(1, K - 64), K]
    f0, amps, want, sr = _exact_phases(K, counts, spectrum, 4, 8192, K)
    one = torch.ones(1, 4, device="cuda")
    got = ctx.harmonic_render(f0.cuda(), one, amps.cuda(), one, 8192, sr, phase_mode=dgen_b200.PHASE_FUNDAMENTAL)
    err = [_norm_error(got[b].cpu().double().numpy(), want[b]) for b in range(4)]
    print("K %d %s: %s" % (K, spectrum, " ".join("%.2e" % e for e in err)))
    assert max(err) < PER_PARTIAL


@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 7, 8, 9, 11, 12, 13, 16, 17, 20, 21, 24, 28, 100, 128])
def test_few_audible_partials(ctx, K):
    """Rows of few partials and rows of many of which few are heard: at the edges of fours, eights, of the count that a warp takes
    partial by partial and of the row lengths that always are."""
    counts = [c for c in (1, 2, 3, 4, 5, 7, 8, 9, 12, 13, 16, 17, 20, 24) if c < K] + [K, K]
    f0, amps, want, sr = _exact_phases(K, counts, "flat", len(counts), 4097, 100 + K)
    for b, c in enumerate(counts):
        amps[0, b, c:] = float("nan")           # what is not audible is not to come in
    one = torch.ones(1, len(counts), device="cuda")
    got = ctx.harmonic_render(f0.cuda(), one, amps.cuda(), one, 4097, sr, phase_mode=dgen_b200.PHASE_FUNDAMENTAL).cpu().double()
    for b, c in enumerate(counts):
        assert _norm_error(got[b].numpy(), want[b]) < PER_PARTIAL, c


def test_counts_that_change_inside_a_warp(ctx):
    """f0 sweeps the audible count of 100 partials from 100 to 1 and back within a few hundred frames: warps on both sides of the
    rule and across it."""
    g = torch.Generator().manual_seed(3)
    f0 = torch.tensor([79.0, 8000.0 / 6, 7000.0, 900.0, 1000.0, 8000.0 / 9])[:, None].repeat(1, 2)
    amps = torch.rand(6, 2, 100, generator=g)
    got = _render(ctx, f0, amps, 640).cpu().double()
    assert (got - _double(f0, amps, 640)).abs().max() < 1e-6 + 2 * np.pi * 100 * 640 * 2.0 ** -33


@pytest.mark.parametrize("K", [5, 12, 60, 130])
def test_a_plan_step_and_the_direct_call(ctx, K):
    """The step without a scratch is the direct call, bit for bit, whether that is given one or not; with one, a training step's, it
    takes a fast sine per partial: the same audio, and the same gradient from the sums left there, to that sine's error."""
    B, T, F = 2, 3000, 40
    hp = dgen_b200.HarmonicParams(B, T, K, F, SR, 1.0, dgen_b200.PHASE_FUNDAMENTAL, 0)
    g = torch.Generator(device="cuda").manual_seed(K)
    draw = lambda lo, hi, *s: torch.rand(*s, generator=g, device="cuda") * (hi - lo) + lo
    ins = [draw(60.0, 400.0, F, B), draw(0.5, 1.0, F, B), draw(0.0, 1.0, F, B, K), draw(0.5, 1.0, F, B)]
    n_scr = int(ctx.lib.dgc_harmonic_bwd_scratch_floats(C.byref(hp)))
    n = [t.numel() for t in ins] + [n_scr, B * T]
    off = [int(o) for o in np.concatenate([[0], np.cumsum([(v + 63) // 64 * 64 for v in n])])]
    arena = torch.zeros(off[-1], device="cuda")
    for o, t in zip(off, ins):
        arena[o:o + t.numel()] = t.reshape(-1)
    h = C.c_void_p()
    ctx.check(ctx.lib.dgc_arena_wrap(ctx.h, arena.data_ptr(), arena.numel(), C.byref(h)))

    def step(scratch):
        a = off[:4] + [off[4] if scratch else None, off[5]]
        steps = (dgen_b200.PlanStep * 1)(dgen_b200.plan_step(dgen_b200.PLAN_HARMONIC_RENDER, a=a,
                                                             i=(B, T, K, F, dgen_b200.PHASE_FUNDAMENTAL, 0), f=(SR, 1.0)))
        plan = dgen_b200.Plan(steps, 1, None, None, 0)
        ctx.check(ctx.lib.dgc_plan_run(ctx.h, h, C.byref(plan), 0, -1))
        ctx.sync()
        return arena[off[5]:off[5] + B * T].view(B, T).clone()

    ga = torch.randn(B, T, generator=g, device="cuda")

    def gradient(scratch_ptr):
        out = torch.empty(F, B, K, device="cuda")
        ctx.check(ctx.lib.dgc_harmonic_render_bwd_prepared(ctx.h, C.byref(hp), *[t.data_ptr() for t in ins], ga.data_ptr(), scratch_ptr,
                                                           out.data_ptr()))
        ctx.sync()
        return out.double()

    scratch = torch.empty(n_scr, device="cuda")
    kw = dict(phase_mode=dgen_b200.PHASE_FUNDAMENTAL)
    direct, kept = ctx.harmonic_render(*ins, T, SR, **kw), ctx.harmonic_render(*ins, T, SR, scratch=scratch, **kw)
    assert torch.equal(direct, kept) and torch.equal(step(False), direct)
    training = step(True)
    assert float((training - direct).double().norm() / direct.double().norm()) < 1e-6
    a, b = gradient(scratch.data_ptr()), gradient(arena.data_ptr() + 4 * off[4])
    assert float((a - b).norm() / b.norm()) < 1e-6
    ctx.lib.dgc_arena_destroy(h)


@pytest.mark.parametrize("K", [1, 4, 12])
def test_few_partials_are_no_slower_than_a_sine_each(ctx, K):
    """The render of a plan step that keeps its scratch takes a fast sine per partial; fewer partials than a group must not take longer
    than that (it also stores the track and its sums, a few per cent)."""
    B, T, F = 256, 64000, 1000
    f0, one = torch.full((F, B), 100.0, device="cuda"), torch.ones(F, B, device="cuda")
    hp = dgen_b200.HarmonicParams(B, T, K, F, SR, 1.0, dgen_b200.PHASE_FUNDAMENTAL, 0)
    n = [F * B, F * B, F * B * K, F * B, int(ctx.lib.dgc_harmonic_scratch_floats(C.byref(hp))), B * T]
    off = np.concatenate([[0], np.cumsum([(v + 63) // 64 * 64 for v in n])])
    arena = torch.zeros(int(off[-1]), device="cuda")
    arena[:n[0]] = 100.0
    for i in (1, 3):
        arena[off[i]:off[i] + n[i]] = 1.0
    amps = arena[off[2]:off[2] + n[2]].uniform_()
    steps = (dgen_b200.PlanStep * 1)(dgen_b200.plan_step(dgen_b200.PLAN_HARMONIC_RENDER, a=[int(o) for o in off[:6]],
                                                         i=(B, T, K, F, dgen_b200.PHASE_FUNDAMENTAL, 0), f=(SR, 1.0)))
    plan = dgen_b200.Plan(steps, 1, None, None, 0)
    h = C.c_void_p()
    ctx.check(ctx.lib.dgc_arena_wrap(ctx.h, arena.data_ptr(), arena.numel(), C.byref(h)))
    out = torch.empty(B, T, device="cuda")
    calls = (lambda: ctx.harmonic_render(f0, one, amps.view(F, B, K), one, T, SR, phase_mode=dgen_b200.PHASE_FUNDAMENTAL, out=out),
             lambda: ctx.check(ctx.lib.dgc_plan_run(ctx.h, h, C.byref(plan), 0, -1)))
    times = ([], [])
    for rep in range(13):
        for call, ts in zip(calls, times):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            call()
            b.record()
            torch.cuda.synchronize()
            if rep >= 3:
                ts.append(a.elapsed_time(b))
    ctx.lib.dgc_arena_destroy(h)
    groups, sines = (sorted(ts)[len(ts) // 2] for ts in times)
    print("K %d: %.1f us, a sine each %.1f us" % (K, 1e3 * groups, 1e3 * sines))
    assert torch.allclose(out, arena[off[5]:off[5] + n[5]].view(B, T), atol=2e-6)
    assert groups < 1.02 * sines
