"""Tile occlusion in binning and the depth-order-free tile lists: pairs hidden behind a triangle
that covers their tile are dropped, and the frame is what the oracle renders, bit for bit in
depth and stencil, for every state that qualifies and beside every state that must not."""
import ctypes

import numpy as np
import pytest

import harness
from mytinygl_gb300 import gl as G
from mytinygl_gb300.scene import Scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    return harness.product()


@pytest.fixture(scope="module")
def oracle():
    return harness.oracle()


SIZES = [(1, 1), (16, 16), (15, 17), (33, 31), (64, 48), (161, 130), (520, 300)]
STATES = ["less", "lequal", "ties_less", "ties_lequal", "mixed_funcs", "scissor", "depth_range", "greater_after",
          "always_between", "no_write_after", "mask_none", "mask_part", "blend", "stencil", "lines", "alpha_textured",
          "flat", "cleared_near", "nan_clear"]


def _layer(s, rng, n, zlo, zhi, spread, slope=0.05):
    """n triangles around the view (identity transforms), from slivers to ones covering all of it."""
    c = rng.uniform(-1.2, 1.2, (n, 1, 2))
    o = rng.uniform(-1, 1, (n, 3, 2)) * np.exp(rng.uniform(np.log(0.02), np.log(spread), (n, 1, 1)))
    z = rng.uniform(zlo, zhi, (n, 1, 1)) + rng.uniform(-slope, slope, (n, 3, 1))
    pos = np.ascontiguousarray(np.concatenate([c + o, z], 2).reshape(-1, 3).astype(np.float32))
    col = rng.integers(0, 256, (3 * n, 4), dtype=np.uint8)
    s.glVertexPointer(3, G.GL_FLOAT, 0, pos)
    s.glColorPointer(4, G.GL_UNSIGNED_BYTE, 0, col)
    s.glDrawArrays(G.GL_TRIANGLES, 0, 3 * n)


def _quads(s, rng, depths):
    """Screen-covering quads at the given depths, each its own colour (equal depths tie)."""
    pos, col = [], []
    for z in depths:
        pos += [(-1.1, -1.1, z), (1.1, -1.1, z), (1.1, 1.1, z), (-1.1, 1.1, z)]
        col += [rng.integers(0, 256, 4)] * 4
    pos, col = np.array(pos, np.float32), np.array(col, np.uint8)
    s.glVertexPointer(3, G.GL_FLOAT, 0, pos)
    s.glColorPointer(4, G.GL_UNSIGNED_BYTE, 0, col)
    s.glDrawArrays(G.GL_QUADS, 0, len(pos))


def scene(state, w, h):
    rng = np.random.default_rng([w, h, STATES.index(state)])
    s = Scene(f"occlusion_{state}_{w}x{h}", w, h)
    s.glGenTextures(1, np.zeros(1, np.uint32))
    s.glBindTexture(G.GL_TEXTURE_2D, 1)
    s.glTexImage2D(G.GL_TEXTURE_2D, 0, G.GL_RGBA, 8, 8, 0, G.GL_RGBA, G.GL_UNSIGNED_BYTE,
                   rng.integers(0, 256, (8, 8, 4), dtype=np.uint8))
    s.glViewport(0, 0, w, h)
    if state == "cleared_near":
        s.glClearDepth(0.3)
    if state == "nan_clear":
        s.glClearDepth(float("nan"))
    s.glClear(G.GL_COLOR_BUFFER_BIT | G.GL_DEPTH_BUFFER_BIT | G.GL_STENCIL_BUFFER_BIT)
    s.glEnable(G.GL_DEPTH_TEST)
    s.glDepthFunc(G.GL_LEQUAL if "lequal" in state else G.GL_LESS)
    s.glShadeModel(G.GL_FLAT if state == "flat" else G.GL_SMOOTH)
    for a in (G.GL_VERTEX_ARRAY, G.GL_COLOR_ARRAY):
        s.glEnableClientState(a)
    _layer(s, rng, 120, -0.9, 0.9, 1.5)
    if state.startswith("ties"):
        _quads(s, rng, [0.5, 0.25, 0.25, 0.25, 0.5, 0.25])
    _quads(s, rng, [0.6, -0.1, 0.2])
    if state == "mixed_funcs":
        s.glDepthFunc(G.GL_LEQUAL)
        _quads(s, rng, [-0.1, -0.1])
        s.glDepthFunc(G.GL_LESS)
        _quads(s, rng, [-0.1])
    if state == "scissor":
        s.glEnable(G.GL_SCISSOR_TEST)
        s.glScissor(w // 5, h // 7, max(1, w // 2), max(1, h // 2))
        _quads(s, rng, [-0.7])
        s.glDisable(G.GL_SCISSOR_TEST)
    if state == "depth_range":
        s.glDepthRange(0.8, 0.1)
        _layer(s, rng, 40, -0.9, 0.9, 1.5)
        s.glDepthRange(0.0, 1.0)
    if state == "greater_after":
        s.glDepthFunc(G.GL_GREATER)
        _quads(s, rng, [0.4])
        s.glDepthFunc(G.GL_LESS)
    if state == "always_between":
        s.glDepthFunc(G.GL_ALWAYS)
        _layer(s, rng, 10, -0.9, 0.9, 1.5)
        s.glDepthFunc(G.GL_LESS)
    if state == "no_write_after":
        s.glDepthMask(0)
        _layer(s, rng, 40, -0.9, 0.9, 1.5)
        s.glDepthMask(1)
    if state == "mask_none":
        s.glColorMask(0, 0, 0, 0)
        _quads(s, rng, [-0.4])
        s.glColorMask(1, 1, 1, 1)
    if state == "mask_part":
        s.glColorMask(1, 0, 1, 0)
        _quads(s, rng, [-0.4])
        s.glColorMask(1, 1, 1, 1)
    if state == "blend":
        s.glEnable(G.GL_BLEND)
        s.glBlendFunc(G.GL_SRC_ALPHA, G.GL_ONE_MINUS_SRC_ALPHA)
        _quads(s, rng, [-0.4])
        s.glDisable(G.GL_BLEND)
    if state == "stencil":
        s.glEnable(G.GL_STENCIL_TEST)
        s.glStencilFunc(G.GL_ALWAYS, 1, 0xFF)
        s.glStencilOp(G.GL_KEEP, G.GL_INCR, G.GL_REPLACE)
        _quads(s, rng, [-0.3])
        s.glDisable(G.GL_STENCIL_TEST)
    if state == "lines":
        _layer(s, rng, 4, -0.9, 0.9, 1.5)
        s.glPolygonMode(G.GL_FRONT_AND_BACK, G.GL_LINE)
        _layer(s, rng, 20, -0.9, 0.9, 1.5)
        s.glPolygonMode(G.GL_FRONT_AND_BACK, G.GL_FILL)
    if state == "alpha_textured":
        s.glEnable(G.GL_TEXTURE_2D)
        s.glTexCoord2f(0.4, 0.6)
        s.glEnable(G.GL_ALPHA_TEST)
        s.glAlphaFunc(G.GL_GREATER, 0.99)  # discards: the quad hides nothing
        _quads(s, rng, [-0.5])
        s.glDisable(G.GL_ALPHA_TEST)
        s.glDisable(G.GL_TEXTURE_2D)
    _layer(s, rng, 150, -0.9, 0.9, 1.5)
    _quads(s, rng, [-0.2, 0.1])
    _layer(s, rng, 60, -0.95, 0.9, 0.3, slope=0.5)
    return s


@pytest.mark.parametrize("state", STATES)
def test_hidden_pairs_change_nothing(gpu, oracle, state):
    from mytinygl_gb300.scene import render

    gpu.lib.mtgl_set_option.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int]
    for w, h in SIZES:
        s = scene(state, w, h)
        want = render(oracle, s)
        outs = []
        for rejection in (1, 0):  # with the depth rejection off nothing is dropped
            ctx = gpu.context(w, h)
            assert gpu.lib.mtgl_set_option(ctx.handle, 1, rejection) == 0
            s.play(ctx)
            outs.append(ctx.read() + (ctx.glGetError(),))
            ctx.destroy()
        harness.assert_parity(harness.compare(outs[0], outs[1]), color_tol=0, name=f"{s.name} on/off")
        harness.assert_parity(harness.compare(want, outs[0]), color_tol=1, name=s.name)


@pytest.mark.parametrize("tile_size", [8, 16, 32])
def test_hidden_pairs_in_a_batch(gpu, tile_size):
    """Frames that qualify beside frames that do not, at every tile size, against the plain path."""
    scenes = [scene(st, w, h) for st, (w, h) in zip(STATES, SIZES * 3)]
    plain = []
    for s in scenes:
        ctx = gpu.context(s.width, s.height)
        s.play(ctx)
        plain.append(ctx.read())
        ctx.destroy()
    ctxs = [gpu.context(s.width, s.height) for s in scenes]
    for c, s in zip(ctxs, scenes):
        s.play(c, 0, 3)  # the texture
    batch = gpu.batch(tile_size=tile_size)
    for _ in range(2):
        for c, s in zip(ctxs, scenes):
            s.play(c, 3)
        batch.render(ctxs)
        batch.wait()
        for c, s, want in zip(ctxs, scenes, plain):
            got = c.read()
            harness.assert_parity(harness.compare(want + (0,), got + (0,)), color_tol=0, name=f"{s.name} batched")
    batch.destroy()
    for c in ctxs:
        c.destroy()


@pytest.mark.parametrize("rule", ["no_depth", "no_depth_then_depth", "always", "always_no_write", "equal_ties"])
def test_last_fragment_wins_without_a_depth_order(gpu, oracle, rule):
    """Frames decided by submission order alone (no depth test, or one that always passes), and
    coplanar layers decided by it: records are made in any order, the frame is the oracle's."""
    from mytinygl_gb300.scene import render

    for w, h in SIZES:
        rng = np.random.default_rng([w, h, 77])
        s = Scene(f"{rule}_{w}x{h}", w, h)
        s.glViewport(0, 0, w, h)
        s.glClear(G.GL_COLOR_BUFFER_BIT | G.GL_DEPTH_BUFFER_BIT | G.GL_STENCIL_BUFFER_BIT)
        for a in (G.GL_VERTEX_ARRAY, G.GL_COLOR_ARRAY):
            s.glEnableClientState(a)
        if not rule.startswith("no_depth"):
            s.glEnable(G.GL_DEPTH_TEST)
        s.glDepthFunc({"equal_ties": G.GL_LEQUAL}.get(rule, G.GL_ALWAYS if "always" in rule else G.GL_LESS))
        if rule == "always_no_write":
            s.glDepthMask(0)
        _layer(s, rng, 300, -1.2, 1.2, 1.5, slope=0.0 if rule == "equal_ties" else 0.4)
        _quads(s, rng, [0.3, 0.3])
        _layer(s, rng, 300, 0.3, 0.3, 1.5, slope=0.0)
        if rule == "no_depth_then_depth":
            s.glEnable(G.GL_DEPTH_TEST)
            _layer(s, rng, 50, -0.9, 0.9, 1.5)
        harness.assert_parity(harness.compare(render(oracle, s), render(gpu, s)), color_tol=1, name=s.name)


@pytest.mark.parametrize("ntri", [1, 31, 16384, 16385, 40000])
def test_straddling_triangles_at_the_clip_launch_boundary(gpu, oracle, ntri):
    """Passes up to 16384 triangles clip in the set-up launch, larger ones in their own."""
    from mytinygl_gb300 import workloads as W
    from mytinygl_gb300.scene import render

    s = W.textured_scene(96, 64, ntri=ntri, seed=ntri, tex_size=16, spread=1.2)
    harness.assert_parity(harness.compare(render(oracle, s), render(gpu, s)), color_tol=1, name=s.name)
