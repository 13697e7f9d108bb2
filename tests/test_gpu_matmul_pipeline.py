"""The tensor-core matmul pipeline with A in tensor memory at the edges of its tiles and of its persistent walk: rows, columns and
reductions that fill no tile, more tiles than CTAs, fewer k tiles than stages, split reductions in both tile widths."""
import numpy as np
import pytest
import torch

import dgen_b200

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = dgen_b200.Context(0)
    yield c
    c.close()


def _tol(n):
    """Three TF32 products leave out lo * lo and what lo loses by truncation, 2^-20 of a term; the accumulator is truncated at each
    of 3 n / 8 steps, 2^-24 of the sum so far (a long reduction is cut into slices of 2048 or less, added in single precision)."""
    return 2.0 ** -20 + 3 * min(n, 2048) / 8 * 2.0 ** -24


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


# (M, K, N): from 149 output tiles of 64 x 64 on and 2^21 products the pipeline takes the layer's three matmuls
@pytest.mark.parametrize("M,K,N,act", [(1000, 32, 640, 0), (1537, 36, 513, 1), (5000, 100, 260, 1), (9600, 512, 128, 0),
                                       (20001, 48, 128, 1), (19000, 68, 132, 0), (24004, 256, 300, 1)])
def test_layers_that_fill_no_tile(ctx, M, K, N, act):
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    a = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randn(K, N, device="cuda", generator=g) * K ** -0.5
    b = torch.randn(N, device="cuda", generator=g)
    c, ct = ctx.linear_fwd(a, w, b, act=act, want_transposed=True)
    z = a.double() @ w.double() + b.double()
    want = torch.tanh(z) if act else z
    assert _rel(c, want) < _tol(K) and torch.equal(ct.t(), c)
    dc = torch.randn(M, N, device="cuda", generator=g)
    dz = dc.double() * (1 - c.double() ** 2) if act else dc.double()
    da, dw, db = ctx.linear_bwd(a, w, c, dc, act=act, a_t=a.t().contiguous())
    assert _rel(da, dz @ w.double().t()) < _tol(N)
    assert _rel(dw, a.double().t() @ dz) < _tol(M)
    assert _rel(db, dz.sum(0)) < _tol(M)
    again, _, _ = ctx.linear_bwd(a, w, c, dc, act=act, a_t=a.t().contiguous())
    assert torch.equal(again, da)
    ctx.sync()


# N not a multiple of 4: the input gradient reads copies of dZ and W in aligned rows (but for few tiles, the second case, and
# a short reduction over 128 columns, the third)
@pytest.mark.parametrize("M,K,N,act", [(4000, 512, 165, 0), (1024, 300, 61, 1), (8000, 130, 70, 0), (9604, 65, 33, 1),
                                       (20000, 100, 35, 0), (5000, 257, 127, 1), (32000, 36, 18, 0)])
def test_input_gradient_of_unaligned_rows(ctx, M, K, N, act):
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    a = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randn(K, N, device="cuda", generator=g) * K ** -0.5
    b = torch.randn(N, device="cuda", generator=g)
    c = ctx.linear_fwd(a, w, b, act=act)
    dc = torch.randn(M, N, device="cuda", generator=g)
    dz = dc.double() * (1 - c.double() ** 2) if act else dc.double()
    at = a.t().contiguous()
    ctx.linear_bwd(a, w, c, torch.full_like(dc, float("nan")), act=act, a_t=at)   # what an earlier call leaves between the rows
    da, dw, db = ctx.linear_bwd(a, w, c, dc, act=act, a_t=at)
    assert _rel(da, dz @ w.double().t()) < _tol(N)
    assert _rel(dw, a.double().t() @ dz) < _tol(M)
    assert _rel(db, dz.sum(0)) < _tol(M)


def test_rows_past_the_end_are_not_read(ctx):
    """NaN behind the operand and in front of it: what the copy engine brings past the last row or column arrives as zeros."""
    M, K, N = 4100, 132, 300
    room = torch.full((M * K + 4096,), float("nan"), device="cuda")
    room[2048:2048 + M * K] = torch.randn(M * K, device="cuda")
    a = room[2048:2048 + M * K].view(M, K)
    w = torch.randn(K, N, device="cuda") * K ** -0.5
    c = ctx.linear_fwd(a, w)
    assert torch.isfinite(c).all() and _rel(c, a.double() @ w.double()) < _tol(K)
    # the operand's own values that are not finite stay in their rows
    a[7, 3] = float("inf")
    c2 = ctx.linear_fwd(a, w)
    rows = torch.isfinite(c2).all(1)
    assert not bool(rows[7]) and int(rows.sum()) == M - 1 and torch.equal(c2[rows], c[rows])


@pytest.mark.parametrize("M", [65535 * 64 - 64, 65535 * 64])
def test_input_gradient_of_unaligned_rows_at_the_edge_of_the_grid(ctx, M):
    """The blocks that copy dZ and those that copy W together are one more than a grid's second dimension holds (the second case)."""
    K, N = 64, 33
    if torch.cuda.mem_get_info()[0] < 12 << 30:
        pytest.skip("12 GB of device memory")
    g = torch.Generator(device="cuda").manual_seed(K + N)
    a = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randn(K, N, device="cuda", generator=g) * K ** -0.5
    dc = torch.randn(M, N, device="cuda", generator=g)
    da, dw, db = ctx.linear_bwd(a, w, None, dc, act=0, a_t=a.t().contiguous())
    for lo in (0, M // 2, M - 1000):
        assert _rel(da[lo:lo + 1000], dc[lo:lo + 1000].double() @ w.double().t()) < _tol(N)
    # one output tile, so as many slices of the rows as two blocks an SM: M / 296 rows each (more, on fewer SMs)
    slices = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    assert _rel(dw, a.double().t() @ dc.double()) < 2.0 ** -20 + 3 * (M / slices) / 8 * 2.0 ** -24
    # sums of 1024 rows by eight threads, then 4096 of those one after the other
    assert _rel(db, dc.double().sum(0)) < (128 + 4096) * 2.0 ** -24
    ctx.sync()


def test_input_gradient_of_unaligned_rows_without_room_for_the_copies():
    """Device memory that holds dZ transposed but not the aligned copies beside it: the layer goes on without them."""
    M, K, N = 400000, 64, 165
    ctx = dgen_b200.Context(0)
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randn(K, N, device="cuda", generator=g) * K ** -0.5
    dc = torch.randn(M, N, device="cuda", generator=g)
    at = a.t().contiguous()
    dz, da, dw, db = dc.clone(), torch.empty_like(a), torch.empty_like(w), torch.empty(N, device="cuda")
    call = lambda da_ptr: ctx.check(ctx.lib.dgc_linear_bwd(ctx.h, a.data_ptr(), w.data_ptr(), None, dc.data_ptr(), M, K, N, 0, dz.data_ptr(),
                                                           da_ptr, dw.data_ptr(), db.data_ptr(), at.data_ptr()))
    call(None)                      # dZ transposed, and the scratch of everything else
    ctx.sync()
    torch.cuda.empty_cache()
    spare, blocks = M * N * 2, []   # half of dZ; with dZ itself given back, one and a half: the call with copies wants two
    while True:
        free = torch.cuda.mem_get_info()[0] - spare
        if free < 4 << 20:
            break
        blocks.append(torch.empty(min(free // (2 << 20) * (2 << 20), 8 << 30), dtype=torch.uint8, device="cuda"))
    try:
        call(da.data_ptr())
        ctx.sync()
        left = torch.cuda.mem_get_info()[0]
        call(da.data_ptr())         # and does not ask again
        assert torch.cuda.mem_get_info()[0] == left
        ctx.sync()
    finally:
        del blocks
        torch.cuda.empty_cache()
    for lo in (0, M // 2, M - 1000):
        assert _rel(da[lo:lo + 1000], dc[lo:lo + 1000].double() @ w.double().t()) < _tol(N)
    ctx.close()
    ctx = dgen_b200.Context(0)
    da2, _, _ = ctx.linear_bwd(a, w, None, dc, act=0, a_t=at)
    assert torch.equal(da2, da)     # with them the same bits
    ctx.close()
