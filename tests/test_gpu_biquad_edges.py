"""The biquad bank where its sweeps change pace: last chunks of one frame, of whole and of broken groups of sixteen, warps with
lanes of edge chunks and of others, runs of chunks just below, at and above the carry's sixteen."""
import numpy as np
import pytest
import torch

import dgen_b200
from dgen_b200 import workloads as wl
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
f32 = np.float32
CHUNK = 512


@pytest.fixture(scope="module")
def ctx():
    c = dgen_b200.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("L,T", [(3, CHUNK + 1), (33, 2 * CHUNK + 15), (40, 2 * CHUNK + 16), (5, 3 * CHUNK + 17),
                                 (2, 15 * CHUNK), (2, 16 * CHUNK), (2, 16 * CHUNK + 1), (2, 17 * CHUNK - 1), (3, 33 * CHUNK)])
def test_chunks_and_groups_at_their_edges(ctx, L, T):
    B = 2
    d = wl.biquad_bank_inputs(L + T, B=B, L=L, T=T)
    x, q = d["x"], d["q"]
    cut = np.exp(np.random.default_rng(L).uniform(np.log(400.0), np.log(8000.0), L)).astype(f32)
    want = orc.biquad_bank(x, cut, q)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    X, C_, Q_ = dev(x), dev(cut), dev(q)
    y = ctx.biquad_fwd(X, C_, Q_)
    assert np.abs(y.cpu().numpy().transpose(0, 2, 1) - want).max() < 1e-4 * max(1.0, np.abs(want).max())
    # in two calls with the state carried, cut inside a chunk: the same sequence
    state = torch.zeros(B, 4, L, device="cuda")
    k = T // 2 + 3
    parts = [ctx.biquad_fwd(X[:, a:b].contiguous(), C_, Q_, state=state) for a, b in ((0, k), (k, T))]
    assert float((torch.cat(parts, 1) - y).abs().max()) < 1e-4 * max(1.0, np.abs(want).max())
    target = orc.biquad_bank(x, cut * f32(1.05), q)
    scale = 1.0 / (B * T)
    _, gc64, gq64 = orc.biquad_bank_mse_grad(x, cut, q, target, scale=scale)
    t = dev(target.transpose(0, 2, 1))
    gc, gq, _ = ctx.biquad_mse_bwd(X, C_, Q_, y, t, loss_scale=scale)
    gy = (2.0 * scale) * (y - t)
    uc, uq, gx = ctx.biquad_bwd(X, C_, Q_, y, gy)
    for got, ref in ((gc, gc64), (gq, gq64), (uc, gc64), (uq, gq64)):
        assert np.abs(got.cpu().numpy() - ref).max() <= 1e-3 * np.abs(ref).max()
    g64 = gy.cpu().numpy().astype(np.float64)
    ref = np.stack([sum(orc.biquad(g64[b, ::-1, l].copy(), float(cut[l]), float(q[l]), double=True)[::-1] for l in range(L))
                    for b in range(B)])
    assert np.abs(gx.cpu().numpy() - ref).max() <= 1e-3 * max(np.abs(ref).max(), 1e-30)
