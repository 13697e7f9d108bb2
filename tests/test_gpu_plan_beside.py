"""Steps of a plan that the library runs beside each other or in one launch: weight gradients of a layer beside the backward of
the next, a sum and its copy.  What they read and write decides, so the buffers here meet in every way they can."""
import ctypes as C
import re

import numpy as np
import pytest
import torch

import dgen_b200
from dgen_b200 import (PLAN_ADD, PLAN_COPY, PLAN_LINEAR_BWD, PLAN_MSS_LOSS_BWD, PLAN_MSS_LOSS_FWD, PLAN_PARTCONV_BWD, Plan, PlanStep,
                       plan_step, trainer)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = dgen_b200.Context(0)
    yield c
    c.close()


def _run(ctx, arena, steps):
    arr = (PlanStep * len(steps))(*steps)
    plan = Plan(arr, len(steps), None, None, 0)
    h = C.c_void_p()
    ctx.check(ctx.lib.dgc_arena_wrap(ctx.h, arena.data_ptr(), arena.numel(), C.byref(h)))
    ctx.check(ctx.lib.dgc_plan_run(ctx.h, h, C.byref(plan), 0, -1))
    ctx.sync()
    ctx.lib.dgc_arena_destroy(h)


def _recorded(ctx, arena, steps, path):
    """The number of nodes of the plan's recording, and whether any work lies beside other work: two first nodes, or two that
    follow one."""
    arr = (PlanStep * len(steps))(*steps)
    plan = Plan(arr, len(steps), None, None, 0)
    h = C.c_void_p()
    ctx.check(ctx.lib.dgc_arena_wrap(ctx.h, arena.data_ptr(), arena.numel(), C.byref(h)))
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph(keep_graph=True)
    g.enable_debug_mode()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s), ctx.on_stream(s):
        ctx.check(ctx.lib.dgc_plan_run(ctx.h, h, C.byref(plan), 0, -1))
    g.debug_dump(str(path))
    ctx.lib.dgc_arena_destroy(h)
    edges = re.findall(r'"(\w+)"\s*->\s*"(\w+)"', path.read_text())
    nodes = set(re.findall(r'"(graph_\w+_node_\d+)"', path.read_text()))
    before = [a for a, _ in edges]
    return len(nodes), len(nodes - {b for _, b in edges}) > 1 or any(before.count(a) > 1 for a in set(before))


# shared: which buffers the layers have in common ("" none; dz: one dZ for all; act: the second layer's dA lands on the first
# layer's input, which its weight gradient reads; grads: one weight gradient buffer, the last one written stays)
@pytest.mark.parametrize("shared", ["", "dz", "act", "grads"])
@pytest.mark.parametrize("M,H", [(300, 64), (750, 128), (2100, 64)])
def test_layers_backward_as_a_plan(ctx, M, H, shared, tmp_path):
    g = torch.Generator(device="cuda").manual_seed(M + H)
    used = 0

    def take(n):
        nonlocal used
        used += (n + 63) // 64 * 64
        return used - (n + 63) // 64 * 64

    L = 3
    x = [take(M * H) for _ in range(L + 1)]            # inputs of the layers, the last layer's output
    w = [take(H * H) for _ in range(L)]
    d = [take(M * H) for _ in range(L + 1)]            # gradients of x
    dz = [take(M * H) for _ in range(L)]
    dw, db = [take(H * H) for _ in range(L)], [take(H) for _ in range(L)]
    if shared == "dz":
        dz = [dz[0]] * L
    if shared == "act":
        d[1] = x[2]                                    # layer 1's dA on the input of layer 2, whose gradient may still be read
    if shared == "grads":
        dw, db = [dw[0]] * L, [db[0]] * L
    arena = torch.randn(used, device="cuda", generator=g) * 0.3
    for o in x[1:]:
        arena[o:o + M * H].tanh_()
    want = arena.clone()
    view = lambda t, o, *s: t[o:o + int(np.prod(s))].view(*s)
    steps = []
    for l in reversed(range(L)):
        steps.append(plan_step(PLAN_LINEAR_BWD, a=(x[l], w[l], x[l + 1], d[l + 1], dz[l], d[l], dw[l], db[l], None), i=(M, H, H, 1)))
        ctx.check(ctx.lib.dgc_linear_bwd(ctx.h, *[want.data_ptr() + 4 * o for o in (x[l], w[l], x[l + 1], d[l + 1])], M, H, H, 1,
                                         *[want.data_ptr() + 4 * o for o in (dz[l], d[l], dw[l], db[l])], None))
    ctx.sync()
    for _ in range(3):
        got = arena.clone()
        _run(ctx, got, steps)
        assert torch.equal(got, want)
    # all gradients of these sizes run beside the next layer's backward; where they meet its buffers it waits for them
    assert _recorded(ctx, arena.clone(), steps, tmp_path / "layers.dot")[1]
    if not shared:
        z = view(arena, d[L], M, H).double() * (1 - view(arena, x[L], M, H).double() ** 2)
        ref = view(arena, x[L - 1], M, H).double().t() @ z
        assert float((view(want, dw[L - 1], H, H).double() - ref).norm() / ref.norm()) < 1e-5


@pytest.mark.parametrize("n", [1, 255, 1000])
def test_sum_and_its_copy(ctx, n, tmp_path):
    base = torch.randn(4 * 1024, device="cuda")
    # the sum of [0, n) and [1024, ..) at 2048 (or over its first term), then a copy of it elsewhere, on a term, on the upper half of
    # itself, of a part of it; one launch only where it lands apart and is whole
    for src, dst, copy_n, one in ((2048, 3072, n, True), (2048, 0, n, False), (2048, 1024, n, False), (2048, 2048 + n // 2, n, False),
                                  (0, 3072, n, True), (2048, 3072, 1, n == 1)):
        want = base.clone()
        want[src:src + n] = want[0:n] + want[1024:1024 + n]
        defined = torch.ones(base.numel(), dtype=torch.bool, device="cuda")
        if dst < src + copy_n and src < dst + copy_n:
            defined[dst:dst + copy_n] = False      # what a copy leaves where its two ranges meet is not defined
        else:
            want[dst:dst + copy_n] = want[src:src + copy_n].clone()
        steps = [plan_step(PLAN_ADD, a=(0, 1024, src, n)), plan_step(PLAN_COPY, a=(src, dst, copy_n))]
        got = base.clone()
        _run(ctx, got, steps)
        assert torch.equal(got[defined], want[defined]), (src, dst)
        nodes, _ = _recorded(ctx, base.clone(), steps, tmp_path / "sum.dot")
        assert nodes == (1 if one else 2), (src, dst, nodes)


def test_a_copy_beyond_the_arena_leaves_the_sum_before_it(ctx):
    """The step that fails is the copy; the sum before it is enqueued as it would be alone."""
    arena = torch.randn(1024, device="cuda")
    want = arena[0:64] + arena[64:128]
    with pytest.raises(dgen_b200.DgenCudaError, match="step 1.*beyond the arena"):
        _run(ctx, arena, [plan_step(PLAN_ADD, a=(0, 64, 128, 64)), plan_step(PLAN_COPY, a=(128, 1000, 64))])
    ctx.sync()
    assert torch.equal(arena[128:192], want)


# meet: where the loss's buffers meet those of the steps after it ("" nowhere; partial: its sums lie in the gradient; pred: the
# convolution's gradient lands on the signal; cell: the loss's value lies in the impulse response's gradient)
@pytest.mark.parametrize("meet", ["", "partial", "pred", "cell"])
def test_loss_beside_its_gradient(ctx, meet, tmp_path):
    B, T, N, ir = 6, 30000, 256, 1000
    sizes = (512, 128, 64)
    mp = dgen_b200.mss_params(B, T, sizes)
    n_part, bt = int(ctx.lib.dgc_mss_partial_floats(C.byref(mp))), B * T
    off = {}
    used = 0
    for name, n in (("pred", bt), ("target", bt), ("grad", max(bt, n_part)), ("part", n_part), ("loss", 64), ("x", bt), ("ir", ir),
                    ("g_ir", ir), ("gx", bt)):
        off[name] = used
        used += (n + 63) // 64 * 64
    if meet == "partial":
        off["part"] = off["grad"]
    if meet == "pred":
        off["gx"] = off["pred"]
    if meet == "cell":
        off["loss"] = off["g_ir"] + 2
    arena = torch.randn(used, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)) * 0.3
    want = arena.clone()
    p = lambda name: want.data_ptr() + 4 * off[name]
    ctx.check(ctx.lib.dgc_mss_loss_fwd(ctx.h, C.byref(mp), p("pred"), p("target"), p("part"), p("loss")))
    ctx.check(ctx.lib.dgc_mss_loss_bwd(ctx.h, C.byref(mp), p("pred"), p("target"), 1.0, p("grad")))
    ctx.check(ctx.lib.dgc_partconv_bwd(ctx.h, p("x"), B, T, p("ir"), ir, N, N // 2, 1.0, p("grad"), None, 0, p("gx"), p("g_ir")))
    ctx.sync()
    shape = (B, T, len(sizes), mp.hop_div) + sizes
    steps = [plan_step(PLAN_MSS_LOSS_FWD, a=(off["pred"], off["target"], off["part"], off["loss"]), i=shape, f=(mp.w_lin, mp.w_log)),
             plan_step(PLAN_MSS_LOSS_BWD, a=(off["pred"], off["target"], off["grad"]), i=shape, f=(mp.w_lin, mp.w_log, 1.0)),
             plan_step(PLAN_PARTCONV_BWD, a=(off["x"], off["ir"], off["grad"], None, off["gx"], off["g_ir"]),
                       i=(B, T, ir, N, N // 2, 0), f=(1.0,))]
    for _ in range(3):
        got = arena.clone()
        _run(ctx, got, steps)
        assert torch.equal(got, want)
    assert _recorded(ctx, arena.clone(), steps, tmp_path / "loss.dot")[1] == (meet != "partial")
    assert not _recorded(ctx, arena.clone(), steps[:1], tmp_path / "loss.dot")[1]


def test_the_loss_step_of_a_training_plan_runs_by_itself(ctx):
    """A host that changes the audio, or times the steps one by one, runs the loss's step alone."""
    m = trainer.HarmonicModel(ctx, 2, 4000, K=12, F=50, nbands=9, taps=33, hidden=32, ir_len=300, conv_n=256, conv_hop=128, sizes=(512, 128))
    g = torch.Generator(device="cuda").manual_seed(2)
    assert m.lay.n_steps == 28
    for v in m.input_views():
        v.copy_(torch.rand(v.shape, device="cuda", generator=g))
    m.forward(*m.input_views())
    ctx.sync()
    want = m.loss.clone()
    assert float(want[0]) > 0.0
    m.loss.zero_()
    m._run(m.i_backward - 1, 1)
    ctx.sync()
    assert torch.equal(m.loss, want)
    m.close()
