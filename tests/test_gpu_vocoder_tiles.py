"""The phase vocoder at the edges of its tiles of 32 hops and 32 bins and of its runs of eight hops, in one call and cut in two."""
import numpy as np
import pytest
import torch

import dgen_b200
from oracle import stateful_ops as so

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.fixture(scope="module")
def ctx():
    c = dgen_b200.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("H,N,hop", [(1, 32, 8), (2, 33, 8), (7, 64, 16), (9, 96, 24), (31, 64, 16), (32, 40, 10), (33, 64, 16),
                                     (64, 64, 16), (65, 70, 16), (97, 64, 16)])
def test_tiles_of_hops_and_bins(ctx, H, N, hop):
    rng = np.random.default_rng(H * 100 + N)
    V = 2
    # every bin well above rounding: the phase of a bin with hardly any energy is decided by it
    mag, arg = rng.uniform(0.5, 2.0, (V, H, N)), rng.uniform(-np.pi, np.pi, (V, H, N))
    re, im = (mag * np.cos(arg)).astype(f32), (mag * np.sin(arg)).astype(f32)
    ratio = rng.uniform(0.6, 1.5, (V, H)).astype(f32)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    got = ctx.phase_vocoder(dev(re), dev(im), dev(ratio), hop)
    again = ctx.phase_vocoder(dev(re), dev(im), dev(ratio), hop)
    assert torch.equal(got[0], again[0]) and torch.equal(got[1], again[1])
    state = torch.zeros(V, 2 * N + 1, device="cuda")
    k = max(1, H // 2)
    parts = [ctx.phase_vocoder(dev(re[:, a:b]), dev(im[:, a:b]), dev(ratio[:, a:b]), hop, state=state)
             for a, b in ((0, k), (k, H)) if b > a]
    for v in range(V):
        w_re, w_im, _ = so.phase_vocoder(re[v], im[v], ratio[v], hop)
        # a phase is a sum of H terms of up to hop pi: their rounding, and that of a sine
        tol = 2.0 * (2e-6 + H * hop * np.pi * 2.0 ** -23)
        for i, want in enumerate((w_re, w_im)):
            assert np.abs(got[i][v].cpu().numpy() - want).max() < tol
            cut = torch.cat([p[i] for p in parts], 1)[v].cpu().numpy()
            assert np.abs(cut - want).max() < tol
    assert bool((state[:, N:2 * N].abs() <= np.pi + 1e-6).all())


@pytest.mark.parametrize("N,hop", [(2048, 2048), (1024, 512)])
def test_a_stream_in_parts_is_the_same_bits_as_in_one(ctx, N, hop):
    """High bins advance by hundreds of turns a hop, and counting them is now and then one off: the phase that a call hands on has
    to be the one that the next hop would have gone on from."""
    rng = np.random.default_rng(N)
    V, H, cuts = 8, 13, (0, 1, 3, 4, 6, 9, 12, 13)
    re, im = (torch.from_numpy(rng.standard_normal((V, H, N)).astype(f32)).cuda() for _ in range(2))
    ratio = torch.from_numpy(rng.uniform(0.7, 1.4, (V, H)).astype(f32)).cuda()
    whole = torch.zeros(V, 2 * N + 1, device="cuda")
    want = ctx.phase_vocoder(re, im, ratio, hop, state=whole)
    state = torch.zeros(V, 2 * N + 1, device="cuda")
    parts = [ctx.phase_vocoder(re[:, a:b].contiguous(), im[:, a:b].contiguous(), ratio[:, a:b].contiguous(), hop, state=state)
             for a, b in zip(cuts, cuts[1:])]
    for i in range(2):
        assert torch.equal(torch.cat([p[i] for p in parts], 1), want[i])
    assert torch.equal(state, whole)
    assert bool((state[:, N:2 * N].abs() <= float(f32(np.pi))).all())
