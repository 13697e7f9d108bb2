"""The harmonic render in groups of eight partials, where its grouping can go wrong: fewer partials than a group, one more or
one less than whole groups, rows that no 16-byte load fits, counts that change inside a warp, phases at zero and half turns."""
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
