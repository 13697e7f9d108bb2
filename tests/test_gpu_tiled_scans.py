"""Scans whose tiles hand values on inside one launch: sizes around the tile edges, states that live longer than a tile."""
import numpy as np
import pytest
import torch

import dgen_b200
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.fixture(scope="module")
def ctx():
    c = dgen_b200.Context(0)
    yield c
    c.close()


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("B,T,a", [(1, 2047, 0.9), (1, 2048, 0.9), (2, 2049, 0.9), (3, 4097, 0.0), (2, 70003, 0.9999),
                                   (1, 200000, 0.999999), (700, 6000, -0.97)])
def test_onepole_tiles(ctx, B, T, a):
    rng = np.random.default_rng(B + T)
    x = rng.standard_normal((B, T)).astype(f32)
    y0 = rng.standard_normal(B).astype(f32)
    first = x.copy()
    first[:, 0] += f32(a) * y0
    want = np.stack([orc.onepole(first[b].astype(np.float64), a, double=True) for b in range(B)])
    state = dev(y0)
    got = ctx.onepole_fwd(dev(x), a, state=state)
    assert np.abs(got.cpu().numpy() - want).max() <= 1e-5 * max(1.0, np.abs(want).max())
    assert torch.equal(state, got[:, -1])
    assert torch.equal(ctx.onepole_fwd(dev(first), a), ctx.onepole_fwd(dev(first), a))
