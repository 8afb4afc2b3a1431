"""Triangles crossing several clip planes: the passes over planes that a polygon is already
inside are left out, and the polygons match the reference's in every byte."""
import numpy as np
import pytest

import harness
from mytinygl_gb300 import gl as G
from mytinygl_gb300.scene import Scene, render

pytestmark = pytest.mark.gpu


def shards(n, blend, seed):
    """n triangles with corners in and around the view volume, some on its planes."""
    rng = np.random.default_rng([n, blend, seed])
    w, h = 61, 43
    s = Scene("shards", w, h)
    s.glViewport(0, 0, w, h)
    s.glClear(G.GL_COLOR_BUFFER_BIT | G.GL_DEPTH_BUFFER_BIT)
    s.glMatrixMode(G.GL_PROJECTION)
    s.glLoadIdentity()
    s.glFrustum(-1.0, 1.0, -1.0, 1.0, 1.0, 4.0)
    s.glMatrixMode(G.GL_MODELVIEW)
    s.glLoadIdentity()
    s.glEnable(G.GL_DEPTH_TEST)
    s.glDepthFunc(G.GL_LESS)
    if blend:
        s.glEnable(G.GL_BLEND)
        s.glBlendFunc(G.GL_SRC_ALPHA, G.GL_ONE_MINUS_SRC_ALPHA)
    reach = np.where(rng.random((n, 1, 1)) < 0.5, 1.5, 6.0)
    pos = rng.uniform(-1.0, 1.0, (n, 3, 3)) * reach
    pos[:, :, 2] -= 2.5
    on = rng.random((n, 3)) < 0.2  # corners exactly on a side plane, the near or the far one
    pos[on, 0] = pos[on, 2] * rng.choice([-1.0, 1.0], int(on.sum()))
    on = rng.random((n, 3)) < 0.1
    pos[on, 2] = rng.choice([-1.0, -4.0, 0.0], int(on.sum()))
    col = rng.integers(0, 256, (n * 3, 4), dtype=np.uint8)
    s.glEnableClientState(G.GL_VERTEX_ARRAY)
    s.glEnableClientState(G.GL_COLOR_ARRAY)
    s.glVertexPointer(3, G.GL_FLOAT, 0, np.ascontiguousarray(pos.reshape(-1, 3), np.float32))
    s.glColorPointer(4, G.GL_UNSIGNED_BYTE, 0, col)
    s.glDrawArrays(G.GL_TRIANGLES, 0, 3 * n)
    return s


@pytest.mark.parametrize("blend", [0, 1], ids=["any_order", "in_order"])
@pytest.mark.parametrize("n", [1, 33, 400, 6000])
def test_polygons_across_planes(n, blend):
    gpu, oracle = harness.product(), harness.oracle()
    for seed in range(3):
        s = shards(n, blend, seed)
        harness.assert_parity(harness.compare(render(oracle, s), render(gpu, s)), color_tol=0,
                              name=f"{n} {blend} {seed}")
