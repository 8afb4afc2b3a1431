"""Ordered frames whose tiles hold about one, two or three of the tile kernel's chunks of records,
with records that raise depths anywhere in them, match the oracle in every byte."""
import numpy as np
import pytest

import harness
from mytinygl_gb300 import gl as G
from mytinygl_gb300.scene import Scene, render

pytestmark = pytest.mark.gpu

W, H = 37, 21


def layers(n, textured, wide, seed):
    """n blended triangles over one another in a few tiles, in draws of their own depth functions;
    `wide` of them cover the whole frame."""
    rng = np.random.default_rng([n, textured, wide, seed])
    s = Scene("layers", W, H)
    if textured:
        s.glGenTextures(1, np.zeros(1, np.uint32))
        s.glBindTexture(G.GL_TEXTURE_2D, 1)
        s.glTexImage2D(G.GL_TEXTURE_2D, 0, G.GL_RGBA, 8, 8, 0, G.GL_RGBA, G.GL_UNSIGNED_BYTE,
                       rng.integers(0, 256, (8, 8, 4), dtype=np.uint8))
        s.glEnable(G.GL_TEXTURE_2D)
        s.glEnableClientState(G.GL_TEXTURE_COORD_ARRAY)
    s.glViewport(0, 0, W, H)
    s.glClear(G.GL_COLOR_BUFFER_BIT | G.GL_DEPTH_BUFFER_BIT)
    s.glEnable(G.GL_DEPTH_TEST)
    s.glEnable(G.GL_BLEND)
    s.glBlendFunc(G.GL_SRC_ALPHA, G.GL_ONE_MINUS_SRC_ALPHA)
    s.glEnableClientState(G.GL_VERTEX_ARRAY)
    s.glEnableClientState(G.GL_COLOR_ARRAY)
    pos = rng.uniform(-1.0, 1.0, (n, 1, 3)) + rng.uniform(-0.3, 0.3, (n, 3, 3))
    flat = rng.random(n) < 0.5  # equal depths among them, the nearest possible one too
    pos[flat, :, 2] = rng.choice([-1.0, -0.5, 0.0, 0.5], int(flat.sum()))[:, None]
    big = rng.permutation(n)[:wide]
    pos[big, :, :2] = np.array([[-1, -1], [3, -1], [-1, 3]])
    pos[:, :, 2] = np.clip(pos[:, :, 2], -1.0, 1.0)
    col = rng.integers(0, 256, (n * 3, 4), dtype=np.uint8)
    s.glVertexPointer(3, G.GL_FLOAT, 0, np.ascontiguousarray(pos.reshape(-1, 3), np.float32))
    s.glColorPointer(4, G.GL_UNSIGNED_BYTE, 0, col)
    if textured:
        s.glTexCoordPointer(2, G.GL_FLOAT, 0, rng.uniform(0, 2, (3 * n, 2)).astype(np.float32))
    funcs = [G.GL_LESS, G.GL_LEQUAL] if seed == 0 else [G.GL_LESS, G.GL_LEQUAL, G.GL_GREATER, G.GL_ALWAYS, G.GL_NEVER]
    first = 0
    while first < n:
        count = min(n - first, int(rng.integers(1, 40)))
        s.glDepthFunc(int(rng.choice(funcs)))
        s.glDrawArrays(G.GL_TRIANGLES, 3 * first, 3 * count)
        first += count
    return s


@pytest.mark.parametrize("textured", [0, 1], ids=["plain", "textured"])
@pytest.mark.parametrize("n,wide", [(1, 0), (32, 32), (33, 3), (63, 60), (64, 64), (65, 65), (130, 9), (700, 20)])
def test_layers(n, wide, textured):
    gpu, oracle = harness.product(), harness.oracle()
    for seed in range(2):
        s = layers(n, textured, wide, seed)
        harness.assert_parity(harness.compare(render(oracle, s), render(gpu, s)), color_tol=0,
                              name=f"{n} {wide} {textured} {seed}")
