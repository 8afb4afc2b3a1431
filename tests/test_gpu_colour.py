"""The tile kernels' packed colour arithmetic rounds as the reference's scalar operations do:
frames whose colours use no transcendental match the oracle in every byte."""
import numpy as np
import pytest

import harness
from mytinygl_gb300 import gl as G
from mytinygl_gb300 import workloads as W
from mytinygl_gb300.scene import Scene, render

pytestmark = pytest.mark.gpu


def quads(w, h, env, blend, mag, min_, wrap, hint=False):
    """Overlapping textured, shaded, fogged quads from magnified to minified, blended."""
    rng = np.random.default_rng([w, h, env, blend[0], blend[1], mag, min_, wrap])
    s = Scene("colour", w, h)
    s.glGenTextures(1, np.zeros(1, np.uint32))
    s.glBindTexture(G.GL_TEXTURE_2D, 1)
    s.glTexImage2D(G.GL_TEXTURE_2D, 0, G.GL_RGBA, 24, 17, 0, G.GL_RGBA, G.GL_UNSIGNED_BYTE,
                   rng.integers(0, 256, (17, 24, 4), dtype=np.uint8))
    s.glTexParameteri(G.GL_TEXTURE_2D, G.GL_TEXTURE_MAG_FILTER, mag)
    s.glTexParameteri(G.GL_TEXTURE_2D, G.GL_TEXTURE_MIN_FILTER, min_)
    s.glTexParameteri(G.GL_TEXTURE_2D, G.GL_TEXTURE_WRAP_S, wrap)
    s.glTexParameteri(G.GL_TEXTURE_2D, G.GL_TEXTURE_WRAP_T, wrap)
    s.glTexEnvi(G.GL_TEXTURE_ENV, G.GL_TEXTURE_ENV_MODE, env)
    s.glTexEnvfv(G.GL_TEXTURE_ENV, G.GL_TEXTURE_ENV_COLOR, np.array([0.3, 0.6, 0.9, 0.7], np.float32))
    s.glViewport(0, 0, w, h)
    s.glClearColor(0.21, 0.43, 0.65, 0.87)
    s.glClear(G.GL_COLOR_BUFFER_BIT | G.GL_DEPTH_BUFFER_BIT)
    s.glEnable(G.GL_TEXTURE_2D)
    s.glEnable(G.GL_FOG)
    s.glFogi(G.GL_FOG_MODE, G.GL_LINEAR)
    s.glFogf(G.GL_FOG_START, -0.9)
    s.glFogf(G.GL_FOG_END, 1.3)
    s.glFogfv(G.GL_FOG_COLOR, np.array([0.5, 0.4, 0.3, 0.6], np.float32))
    if blend[0]:
        s.glEnable(G.GL_BLEND)
        s.glBlendFunc(*blend)
    for k in range(10):
        s.glBegin(G.GL_QUADS)
        c = rng.uniform(-0.9, 0.6, 2)
        size = rng.uniform(0.1, 1.4)
        rep = float(np.exp(rng.uniform(np.log(0.2), np.log(30.0))))
        for x, y in ((0, 0), (1, 0), (1, 1), (0, 1)):
            s.glColor4f(*(float(v) for v in rng.uniform(0, 1, 4)))
            s.glTexCoord2f(rep * x - 0.3, rep * y - 0.2)
            s.glVertex3f(float(c[0] + size * x), float(c[1] + size * y), float(rng.uniform(-0.8, 0.8)))
        s.glEnd()
    return s


BLENDS = [(0, 0), (G.GL_SRC_ALPHA, G.GL_ONE_MINUS_SRC_ALPHA), (G.GL_DST_COLOR, G.GL_ONE_MINUS_SRC_COLOR),
          (G.GL_ONE, G.GL_ONE), (G.GL_SRC_ALPHA_SATURATE, G.GL_DST_ALPHA)]
FILTERS = [(G.GL_NEAREST, G.GL_NEAREST), (G.GL_LINEAR, G.GL_NEAREST_MIPMAP_NEAREST),
           (G.GL_LINEAR, G.GL_LINEAR_MIPMAP_LINEAR), (G.GL_NEAREST, G.GL_LINEAR_MIPMAP_NEAREST),
           (G.GL_NEAREST, G.GL_NEAREST_MIPMAP_LINEAR), (G.GL_LINEAR, G.GL_LINEAR)]


@pytest.mark.parametrize("env", [G.GL_MODULATE, G.GL_REPLACE, G.GL_DECAL, G.GL_BLEND, G.GL_ADD])
def test_textured_colours_are_exact(env):
    gpu, oracle = harness.product(), harness.oracle()
    for k, blend in enumerate(BLENDS):
        for j, (mag, min_) in enumerate(FILTERS):
            wrap = G.GL_REPEAT if (j + k) % 2 else G.GL_CLAMP
            s = quads(97, 61, env, blend, mag, min_, wrap)
            st = harness.compare(render(oracle, s), render(gpu, s))
            # the texture LOD's logarithm moves a blend of two mipmap levels by at most one step
            tol = 1 if min_ in (G.GL_LINEAR_MIPMAP_LINEAR, G.GL_NEAREST_MIPMAP_LINEAR) else 0
            harness.assert_parity(st, color_tol=tol, name=f"{env:#x} {blend} {mag:#x} {min_:#x}")


def test_blended_small_triangles_are_exact():
    gpu, oracle = harness.product(), harness.oracle()
    s = W.rop_scene(333, 222, ntri=30_000)
    harness.assert_parity(harness.compare(render(oracle, s), render(gpu, s)), color_tol=0, name="rop")
