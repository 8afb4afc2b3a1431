"""glTexImage2D from client bytes: every format expanded on the device as the reference packs it,
odd sizes, storage kept across images of one size, and the client's memory free to change."""
import numpy as np
import pytest

import harness
from mytinygl_gb300 import gl as G

pytestmark = pytest.mark.gpu

FORMATS = [(G.GL_RGBA, 4), (G.GL_RGB, 3), (G.GL_LUMINANCE_ALPHA, 2), (G.GL_LUMINANCE, 1)]


def draw(ctx, images):
    """Uploads each image in turn into one texture and draws it minified and magnified."""
    ctx.glViewport(0, 0, 64, 48)
    ctx.glGenTextures(1, np.zeros(1, np.uint32))
    ctx.glBindTexture(G.GL_TEXTURE_2D, 1)
    ctx.glTexParameteri(G.GL_TEXTURE_2D, G.GL_TEXTURE_MIN_FILTER, G.GL_LINEAR_MIPMAP_NEAREST)
    ctx.glEnable(G.GL_TEXTURE_2D)
    ctx.glClear(G.GL_COLOR_BUFFER_BIT | G.GL_DEPTH_BUFFER_BIT | G.GL_STENCIL_BUFFER_BIT)
    for k, (fmt, data) in enumerate(images):
        scratch = data.copy()
        ctx.glTexImage2D(G.GL_TEXTURE_2D, 0, fmt, data.shape[1], data.shape[0], 0, fmt, G.GL_UNSIGNED_BYTE, scratch)
        scratch[:] = 0x5A  # the image was taken during the call
        x = -1.0 + 2.0 * k / len(images)
        for rep, y in ((0.7, -1.0), (9.0, 0.0)):
            ctx.glBegin(G.GL_QUADS)
            for u, v in ((0, 0), (1, 0), (1, 1), (0, 1)):
                ctx.glTexCoord2f(rep * u, rep * v)
                ctx.glVertex2f(x + u * 2.0 / len(images), y + v)
            ctx.glEnd()


@pytest.mark.parametrize("size", [(1, 1), (2, 1), (1, 7), (3, 5), (16, 16), (33, 65), (257, 129)])
def test_formats_and_reuploads(size):
    w, h = size
    rng = np.random.default_rng([w, h])
    images = [(f, rng.integers(0, 256, (h, w, c), dtype=np.uint8)) for f, c in FORMATS + FORMATS[::-1]]
    images.insert(3, (G.GL_RGB, rng.integers(0, 256, (h + 1, w + 2, 3), dtype=np.uint8)))  # another size between
    out = []
    for lib in (harness.oracle(), harness.product()):
        ctx = lib.context(64, 48)
        draw(ctx, images)
        out.append(ctx.read() + (ctx.glGetError(),))
        ctx.destroy()
    harness.assert_parity(harness.compare(*out), color_tol=0, name=f"upload {w}x{h}")
