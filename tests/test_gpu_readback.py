"""Read-backs written by the tile launch: page-locked destinations of a pass that is still queued
(single contexts), and of a batch's larger frames, equal what a later copy gives, in untouched
tiles too; destinations it cannot write are copied."""
import ctypes

import numpy as np
import pytest

import harness
from mytinygl_gb300 import gl as G

pytestmark = pytest.mark.gpu
ALL = G.GL_COLOR_BUFFER_BIT | G.GL_DEPTH_BUFFER_BIT | G.GL_STENCIL_BUFFER_BIT


def triangle(ctx, z, blend):
    (ctx.glEnable if blend else ctx.glDisable)(G.GL_BLEND)
    ctx.glBlendFunc(G.GL_SRC_ALPHA, G.GL_ONE_MINUS_SRC_ALPHA)
    ctx.glEnable(G.GL_DEPTH_TEST)
    ctx.glBegin(G.GL_TRIANGLES)
    for k, (x, y) in enumerate(((-0.7, -0.6), (0.3, -0.5), (-0.1, 0.4))):
        ctx.glColor4f(0.2 + 0.3 * k, 0.9 - 0.2 * k, 0.4, 0.6)
        ctx.glVertex3f(x, y, z)
    ctx.glEnd()


def pinned(torch, n, dtype, off=0):
    t = torch.full((n + 16,), 77, dtype=dtype, pin_memory=True)
    return t, t.data_ptr() + off * t.element_size()


@pytest.mark.parametrize("size", [(1, 1), (17, 9), (64, 48), (131, 257), (640, 360)])
@pytest.mark.parametrize("blend", [False, True], ids=["order-free", "ordered"])
def test_single_context(size, blend):
    torch = pytest.importorskip("torch")
    gpu = harness.product()
    w, h = size
    n = w * h
    ctx = gpu.context(w, h)
    ctx.glViewport(0, 0, w, h)
    read = gpu.lib.mtgl_read_framebuffer
    for case in ("all", "colour", "no clear", "scissored clear", "offset", "pageable depth"):
        if case in ("all", "colour", "offset"):
            ctx.glClear(ALL)
        if case == "scissored clear":
            ctx.glEnable(G.GL_SCISSOR_TEST)
            ctx.glScissor(0, 0, max(1, w // 2), max(1, h // 3))
            ctx.glClear(ALL)
            ctx.glDisable(G.GL_SCISSOR_TEST)
        triangle(ctx, {"all": 0.1, "no clear": -0.2}.get(case, 0.0), blend)
        off = 1 if case == "offset" else 0
        (ct, cp), (dt, dp), (st, sp) = (pinned(torch, n, d, off) for d in (torch.int32, torch.float32, torch.uint8))
        depth = np.full(n, 5.0, np.float32)
        if case == "pageable depth":
            dp = depth.ctypes.data
        args = [cp, dp, sp] if case != "colour" else [cp, None, None]
        assert read(ctx.handle, *(ctypes.c_void_p(a) if a else None for a in args)) == 0
        c, d, s = ctx.read()
        assert np.array_equal(ct.numpy().view(np.uint32)[off:off + n], c.ravel()), case
        assert ct.numpy()[off + n] == 77
        if case != "colour":
            got = depth if case == "pageable depth" else dt.numpy()[off:off + n]
            assert np.array_equal(got, d.ravel()), case
            assert np.array_equal(st.numpy()[off:off + n], s.ravel()), case
            assert st.numpy()[off + n] == 77
    ctx.destroy()


@pytest.mark.parametrize("tile_size", [8, 16, 32])
def test_batch_frames_large_and_small(tile_size):
    """Frames on both sides of the size rule, some without a clear, one rendered twice, and a run
    that exceeds its capacities and is rendered again."""
    torch = pytest.importorskip("torch")
    gpu = harness.product()
    sizes = [(181, 181), (182, 181), (400, 300), (33, 21), (512, 64)]
    ctxs = [gpu.context(w, h) for w, h in sizes]
    b = gpu.batch(tile_size=tile_size, pair_factor=0.01, record_factor=0.01)
    for step in range(3):
        for i, (c, (w, h)) in enumerate(zip(ctxs, sizes)):
            c.make_current()
            c.glViewport(0, 0, w, h)
            if step == 0 or i % 2:
                c.glClear(ALL)
            for k in range(40):
                triangle(c, 0.5 - 0.02 * k - 0.1 * step, blend=(i == 2))
        bufs = [torch.zeros(w * h, dtype=torch.int32, pin_memory=True) for w, h in sizes]
        b.render(ctxs, colors=[t.numpy().view(np.uint32) for t in bufs])
        b.wait()
        for c, t in zip(ctxs, bufs):
            assert np.array_equal(t.numpy().view(np.uint32), c.read()[0].ravel())
    b.destroy()
    for c in ctxs:
        c.destroy()
