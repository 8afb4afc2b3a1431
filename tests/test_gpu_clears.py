"""The clears of a pass, of the whole framebuffer and of parts, in every order, against the oracle."""
import itertools

import numpy as np
import pytest

import harness
from mytinygl_gb300 import gl as G
from mytinygl_gb300.scene import Scene, render

pytestmark = pytest.mark.gpu
C, D, S = G.GL_COLOR_BUFFER_BIT, G.GL_DEPTH_BUFFER_BIT, G.GL_STENCIL_BUFFER_BIT


def frame(w, h, clears, stencil):
    s = Scene("clears", w, h)
    s.glViewport(0, 0, w, h)
    s.glClear(C | D | S)
    s.glEnable(G.GL_DEPTH_TEST)
    for k, (mask, part) in enumerate(clears):
        s.glClearColor(0.1 + 0.2 * k, 0.5, 0.9 - 0.2 * k, 1.0)
        s.glClearDepth(0.9 - 0.2 * k)
        s.glClearStencil(3 + k)
        if part:
            s.glEnable(G.GL_SCISSOR_TEST)
            s.glScissor(w // 4, h // 4, max(1, w // 2), max(1, h // 2))
        s.glClear(mask)
        s.glDisable(G.GL_SCISSOR_TEST)
    if stencil:
        s.glEnable(G.GL_STENCIL_TEST)
        s.glStencilFunc(G.GL_ALWAYS, 0, 0xFF)
        s.glStencilOp(G.GL_KEEP, G.GL_INCR, G.GL_INCR)
    s.glBegin(G.GL_TRIANGLES)
    for x, y in ((-0.9, -0.9), (0.8, -0.7), (0.0, 0.9)):
        s.glVertex3f(x, y, 0.2 + 0.5 * x)
    s.glEnd()
    return s


@pytest.mark.parametrize("size", [(1, 1), (16, 16), (33, 17), (257, 40)])
@pytest.mark.parametrize("stencil", [0, 1])
def test_orders(size, stencil):
    gpu, oracle = harness.product(), harness.oracle()
    kinds = [(C | D, False), (D, False), (S, False), (C | S, True), (D, True)]
    for clears in [()] + [(k,) for k in kinds] + list(itertools.permutations(kinds, 2)) + [tuple(kinds), tuple(kinds[::-1])]:
        s = frame(*size, clears, stencil)
        harness.assert_parity(harness.compare(render(oracle, s), render(gpu, s)), color_tol=0, name=str(clears))
