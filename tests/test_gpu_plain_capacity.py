"""Single-context passes run with capacities learned from earlier passes: a pass beyond them is
rendered again with exact sizes before anything can see its framebuffer or change what it reads."""
import numpy as np
import pytest

import harness
from mytinygl_gb300 import gl as G

pytestmark = pytest.mark.gpu


def quads(ctx, n, seed, w, h):
    """n blended screen-covering quads (many tile pairs per record, in order)."""
    rng = np.random.default_rng(seed)
    ctx.glViewport(0, 0, w, h)
    ctx.glEnable(G.GL_BLEND)
    ctx.glBlendFunc(G.GL_SRC_ALPHA, G.GL_ONE_MINUS_SRC_ALPHA)
    ctx.glBegin(G.GL_QUADS)
    for _ in range(n):
        for x, y in ((-1, -1), (1, -1), (1, 1), (-1, 1)):
            ctx.glColor4f(*(float(v) for v in rng.uniform(0.1, 0.9, 4)))
            ctx.glVertex2f(float(x), float(y))
    ctx.glEnd()


def straddlers(ctx, n, seed):
    """n triangles far larger than the view: each clips to several records."""
    rng = np.random.default_rng(seed)
    ctx.glEnable(G.GL_DEPTH_TEST)
    ctx.glBegin(G.GL_TRIANGLES)
    for _ in range(n):
        a = rng.uniform(0, 2 * np.pi)
        for k in range(3):
            t = a + k * 2 * np.pi / 3
            ctx.glColor3f(*(float(v) for v in rng.uniform(0, 1, 3)))
            ctx.glVertex3f(float(2.5 * np.cos(t)), float(2.5 * np.sin(t)), float(rng.uniform(-3, 3)))
    ctx.glEnd()


ALL = G.GL_COLOR_BUFFER_BIT | G.GL_DEPTH_BUFFER_BIT | G.GL_STENCIL_BUFFER_BIT


def test_pairs_beyond_the_first_estimate():
    """45 screen-covering quads at 1600x1200 make 2^18 tile pairs and more: the first pass runs
    twice, the second (its capacities learned) once, with the same frame."""
    gpu = harness.product()
    ctx = gpu.context(1600, 1200)
    frames, launches = [], []
    for _ in range(2):
        ctx.reset_stats()
        ctx.glClear(ALL)
        quads(ctx, 45, 1, 1600, 1200)
        frames.append(ctx.read() + (ctx.glGetError(),))
        st = ctx.stats()
        assert st["bin_entries"] > 1 << 18 and st["passes"] == 1
        launches.append(st["kernel_launches"])
    assert launches[0] > launches[1]
    harness.assert_parity(harness.compare(*frames), color_tol=0, name="learned capacities")
    ctx.destroy()


@pytest.mark.parametrize("after", ["read", "draw", "clear", "texture", "buffer", "pixels", "flush", "noalloc"])
def test_records_beyond_the_estimate_then(after):
    """300 triangles of several records each, then another operation before the frame is read."""
    out = []
    gpu = harness.product()
    for lib in (harness.oracle(), gpu):
        ctx = lib.context(61, 47)
        ctx.glGenTextures(1, np.zeros(1, np.uint32))
        ctx.glBindTexture(G.GL_TEXTURE_2D, 1)
        tex = np.random.default_rng(3).integers(0, 256, (8, 8, 4), dtype=np.uint8)
        ctx.glTexImage2D(G.GL_TEXTURE_2D, 0, G.GL_RGBA, 8, 8, 0, G.GL_RGBA, G.GL_UNSIGNED_BYTE, tex)
        ctx.glEnable(G.GL_TEXTURE_2D)
        ctx.glTexCoord2f(0.4, 0.6)
        ctx.glViewport(0, 0, 61, 47)
        ctx.glClear(ALL)
        straddlers(ctx, 300, 5)
        ctx.glFlush()
        if after == "draw":
            quads(ctx, 3, 7, 61, 47)
        elif after == "clear":
            ctx.glEnable(G.GL_SCISSOR_TEST)
            ctx.glScissor(10, 8, 20, 20)
            ctx.glClear(ALL)
        elif after == "texture":
            ctx.glTexImage2D(G.GL_TEXTURE_2D, 0, G.GL_RGBA, 8, 8, 0, G.GL_RGBA, G.GL_UNSIGNED_BYTE, 255 - tex)
        elif after == "buffer":
            ctx.glGenBuffers(1, np.zeros(1, np.uint32))
            ctx.glBindBuffer(G.GL_ARRAY_BUFFER, 1)
            ctx.glBufferData(G.GL_ARRAY_BUFFER, 64, np.zeros(64, np.uint8), G.GL_STATIC_DRAW)
        elif after == "pixels":
            ctx.glRasterPos2f(-0.5, -0.5)
            ctx.glDrawPixels(8, 8, G.GL_RGBA, G.GL_UNSIGNED_BYTE, tex)
        elif after == "flush":
            ctx.glFlush()
            straddlers(ctx, 300, 6)
            ctx.glFlush()
        elif after == "noalloc" and lib is gpu:
            assert lib.lib.mtgl_flush_noalloc(ctx.handle) == 0
        out.append(ctx.read() + (ctx.glGetError(),))
        if lib is gpu:
            assert ctx.stats()["setup_triangles"] > 364  # the estimate
        ctx.destroy()
    harness.assert_parity(harness.compare(*out), color_tol=1, name=f"then {after}")


def test_a_batch_settles_its_contexts_first():
    """Contexts with an unchecked pass of their own join a batch, as sources of frames."""
    out = []
    for lib in (harness.oracle(), harness.product()):
        ctxs = [lib.context(61 + 5 * i, 47) for i in range(3)]
        for i, c in enumerate(ctxs):
            c.make_current()
            c.glViewport(0, 0, 61, 47)
            c.glClear(ALL)
            straddlers(c, 300, 5 + i)
            c.glFlush()
            quads(c, 2, i, 61, 47)
        if lib.backend.startswith("cuda"):
            b = lib.batch()
            b.render(ctxs)
            b.wait()
            b.destroy()
        frames = []
        for c in ctxs:
            c.make_current()
            frames.append(c.read() + (c.glGetError(),))
        out.append(frames)
        for c in ctxs:
            c.destroy()
    for i, (a, b) in enumerate(zip(*out)):
        harness.assert_parity(harness.compare(a, b), color_tol=1, name=f"batched after flush {i}")


def test_small_ordered_passes_after_a_large_one():
    """Capacities stay at the largest pass's: passes of no pair, of one, of a few and of many pairs
    (both sides of a sort tile's 2048) follow it in the same context."""
    w, h = 333, 257
    out = []
    for lib in (harness.oracle(), harness.product()):
        ctx = lib.context(w, h)
        ctx.glViewport(0, 0, w, h)
        ctx.glClear(ALL)
        quads(ctx, 900, 11, w, h)
        ctx.glFinish()
        frames = []
        for n, scale in ((0, 1.0), (1, 0.01), (1, 1.0), (6, 1.0), (7, 1.0), (60, 0.3)):
            ctx.glClear(G.GL_COLOR_BUFFER_BIT)
            ctx.glPushMatrix()
            ctx.glScalef(scale, scale, 1.0)
            if n:
                quads(ctx, n, n, w, h)
            else:  # outside the view
                ctx.glTranslatef(5.0, 0.0, 0.0)
                quads(ctx, 3, 3, w, h)
            ctx.glPopMatrix()
            ctx.glFlush()
            frames.append(ctx.read() + (ctx.glGetError(),))
        out.append(frames)
        ctx.destroy()
    for i, (a, b) in enumerate(zip(*out)):
        harness.assert_parity(harness.compare(a, b), color_tol=1, name=f"pass {i}")
