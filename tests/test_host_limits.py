"""What the host does with a pass that fits nowhere or whose memory cannot be had (CPU only: the
library's host code over stand-ins for the CUDA runtime and the kernel launches)."""
import ctypes

import numpy as np
import pytest

import fake_gpu
from mytinygl_gb300 import gl as G

MTGL_OK, MTGL_ERR_OVERFLOW = 0, 7


@pytest.fixture(scope="module")
def fake():
    return fake_gpu.load()


@pytest.fixture
def gpu(fake):
    """(context, controls): a context whose passes make 5 records and 9 pairs."""
    lib, ctl = fake
    ctl.fake_alloc_limit(0)
    ctl.fake_totals(5, 9)
    ctl.fake_log_clear()
    ctx = lib.context(64, 48)
    yield ctx, ctl
    ctl.fake_page_locked(0)
    ctl.fake_alloc_limit(0)
    ctl.fake_totals(5, 9)
    ctx.destroy()


def draw(ctx, triangles=1, blend=False):
    (ctx.glEnable if blend else ctx.glDisable)(G.GL_BLEND)
    ctx.glClear(G.GL_COLOR_BUFFER_BIT)
    ctx.glBegin(G.GL_TRIANGLES)
    for k in range(3 * triangles):
        ctx.glVertex2f(0.1 * (k % 7), 0.1 * (k % 5))
    ctx.glEnd()


def finish(ctx):
    return ctx.glib.lib.mtgl_finish(ctx.handle)


def log(ctl):
    out = ctl.fake_log().decode().split()
    ctl.fake_log_clear()
    return out


@pytest.mark.parametrize("blend", [False, True], ids=["order-free", "ordered"])
def test_totals_past_32_bits_are_refused(gpu, blend):
    """A total that reached the limit of the saturating sums: the capacity run leaves the frame alone,
    the exact one is refused, and the context goes on with its next pass."""
    ctx, ctl = gpu
    for totals in ((5, 0xFFFFFFFF), (0xFFFFFFFF, 0xFFFFFFFF)):
        draw(ctx, blend=blend)
        ctl.fake_totals(*totals)
        assert finish(ctx) == MTGL_ERR_OVERFLOW
        assert "tile" not in log(ctl)
        ctl.fake_totals(5, 9)
        draw(ctx, blend=blend)
        assert finish(ctx) == MTGL_OK and log(ctl)[-1] == "tile"


def test_a_batch_past_32_bits_is_refused(fake, gpu):
    ctx, ctl = gpu
    b = fake[0].batch(use_graph=0)
    draw(ctx)
    ctl.fake_totals(5, 0xFFFFFFFF)
    b.render([ctx])
    assert fake[0].lib.mtgl_dev_batch_wait(b.handle) == MTGL_ERR_OVERFLOW
    assert "tile" not in log(ctl)
    ctl.fake_totals(5, 9)
    draw(ctx)
    b.render([ctx])
    b.wait()
    assert log(ctl)[-1] == "tile"
    b.destroy()


@pytest.mark.parametrize("then", ["nothing", "clear", "draw"])
def test_noalloc_flush_completes_a_flushed_pass_without_allocating(gpu, then):
    """glFlush submits a pass that exceeds its capacities; mtgl_flush_noalloc runs it again, and
    what is queued, from the static array."""
    ctx, ctl = gpu
    for _ in range(2):
        draw(ctx)
        assert finish(ctx) == MTGL_OK
    draw(ctx)
    ctl.fake_totals(5000, 6000)
    ctx.glFlush()
    assert log(ctl)[-1] == "over"
    before = ctl.fake_allocs()
    ctl.fake_totals(6, 10)
    if then == "clear":
        ctx.glClear(G.GL_COLOR_BUFFER_BIT)
    assert ctx.glib.lib.mtgl_flush_noalloc(ctx.handle) == MTGL_OK
    assert log(ctl) == "vertex count emit bin sort tile".split() + ["clear"] * (then == "clear")
    if then == "draw":
        draw(ctx)  # (the draw completes a flushed pass itself)
        before = ctl.fake_allocs()
        assert ctx.glib.lib.mtgl_flush_noalloc(ctx.handle) == MTGL_OK
        assert log(ctl)[-1] == "tile"
    assert ctl.fake_allocs() == before
    assert finish(ctx) == MTGL_OK and ctx.glGetError() == 0


def test_noalloc_flush_refuses_a_flushed_pass_that_does_not_fit(gpu):
    """The flushed pass needs more than the static array: refused, nothing allocated, as often as
    asked, and the next ordinary call renders it."""
    ctx, ctl = gpu
    draw(ctx)
    ctl.fake_totals(400_000, 6000)  # 96 MB of records
    ctx.glFlush()
    log(ctl)
    before = ctl.fake_allocs()
    for _ in range(2):
        assert ctx.glib.lib.mtgl_flush_noalloc(ctx.handle) == MTGL_ERR_OVERFLOW
        assert "tile" not in log(ctl) and ctl.fake_allocs() == before
    assert finish(ctx) == MTGL_OK
    assert log(ctl)[-1] == "tile"
    assert ctx.stats()["setup_triangles"] == 400_000


def draw_many(ctx, n):
    """n triangles over three vertices."""
    pos = np.array([[-0.5, -0.5], [0.5, -0.5], [0.0, 0.5]], np.float32)
    ctx.glClear(G.GL_COLOR_BUFFER_BIT)
    ctx.glEnableClientState(G.GL_VERTEX_ARRAY)
    ctx.glVertexPointer(2, G.GL_FLOAT, 0, pos)
    ctx.glDrawElements(G.GL_TRIANGLES, 3 * n, G.GL_UNSIGNED_INT, np.tile(np.arange(3, dtype=np.uint32), n))


def test_an_estimate_without_memory_takes_exact_sizes(gpu):
    """100,000 triangles of which 5 make records: the estimate asks for 27 MB of records, the pass
    needs 2 MB."""
    ctx, ctl = gpu
    draw_many(ctx, 100_000)
    ctl.fake_alloc_limit(8 << 20)
    ctx.glFlush()
    assert ctx.glGetError() == 0
    assert log(ctl) == "vertex count emit bin sort tile".split()
    assert finish(ctx) == MTGL_OK


def test_a_pass_without_memory_stays_queued(gpu):
    ctx, ctl = gpu
    draw_many(ctx, 1000)
    ctl.fake_alloc_limit(64)
    assert finish(ctx) != MTGL_OK and finish(ctx) != MTGL_OK
    assert "tile" not in log(ctl)
    ctl.fake_alloc_limit(0)
    assert finish(ctx) == MTGL_OK and log(ctl)[-1] == "tile"
    assert ctx.stats()["passes"] == 1


def test_a_second_run_without_memory_is_tried_again(gpu):
    """The pass exceeded its capacities and the exact sizes find no memory: every call that needs the
    frame says so, and the first that finds memory renders it."""
    ctx, ctl = gpu
    draw(ctx)
    ctl.fake_totals(400_000, 6000)
    ctx.glFlush()
    assert log(ctl)[-1] == "over"
    ctl.fake_alloc_limit(8 << 20)
    assert finish(ctx) != MTGL_OK and finish(ctx) != MTGL_OK
    assert "tile" not in log(ctl)
    ctl.fake_alloc_limit(0)
    assert finish(ctx) == MTGL_OK and log(ctl)[-1] == "tile"
    assert ctx.stats()["setup_triangles"] == 400_000


def test_a_failed_read_is_not_written_later(gpu):
    """A read into page-locked memory fails for want of memory: the pass renders later without
    writing that memory."""
    ctx, ctl = gpu
    host = np.zeros(64 * 48, np.uint32)
    read = ctx.glib.lib.mtgl_read_framebuffer
    at = ctypes.c_void_p(host.ctypes.data)
    ctl.fake_page_locked(1)
    draw(ctx)
    assert read(ctx.handle, at, None, None) == MTGL_OK and log(ctl)[-1] == "tile+read"
    draw(ctx)
    ctl.fake_totals(400_000, 6000)
    ctl.fake_alloc_limit(8 << 20)
    assert read(ctx.handle, at, None, None) != MTGL_OK and "over" in log(ctl)
    ctl.fake_alloc_limit(0)
    assert finish(ctx) == MTGL_OK and log(ctl)[-1] == "tile"


def test_a_shared_stream_holds_every_flushed_pass(gpu):
    """A caller that has the context's stream finds a pass that ran twice in it: when it asks for
    the stream after the flush, and when it has it before."""
    ctx, ctl = gpu
    stream = ctx.glib.lib.mtgl_cuda_stream
    stream.argtypes, stream.restype = [ctypes.c_void_p], ctypes.c_void_p
    draw(ctx)
    ctl.fake_totals(5000, 6000)
    ctx.glFlush()
    assert log(ctl)[-1] == "over"
    assert stream(ctx.handle)
    assert log(ctl) == "vertex count emit bin sort tile".split()
    for records in (8000, 9000):
        draw(ctx)
        ctl.fake_totals(records, 6000)
        ctx.glFlush()
        assert log(ctl) == "vertex setup bin over vertex count emit bin sort tile".split()
    draw(ctx)
    ctx.glFlush()
    assert log(ctl) == "vertex setup bin tile".split()


@pytest.mark.parametrize("size,occludes", [((64, 48), 1), ((65536, 2), 1), ((2, 65536), 1), ((65537, 2), 0), ((2, 70000), 0)])
def test_hidden_pairs_are_dropped_where_coordinates_fit(fake, size, occludes):
    """Binning packs pixel coordinates of a record's box into 16 bits to test it against a tile's
    occlusion bound. (gl_create_context stops at 16384; mtgl_dev_create takes any size.)"""
    assert fake[1].fake_occludes(*size) == occludes


@pytest.mark.parametrize("per_sm,side,ctas", [(0, 1024, 64 * 64), (4, 1024, 64 * 64), (3, 1024, 3 * 152), (1, 32, 4)])
def test_batch_stats_count_the_launched_ctas(fake, gpu, per_sm, side, ctas):
    """Tiles of 16 pixels, four CTAs resident per SM of 152: one per tile unless fewer than fit are
    asked for, and never more than tiles."""
    lib = fake[0]
    ctx = lib.context(side, side)
    b = lib.batch(use_graph=0, tile_size=16, ctas_per_sm=per_sm)
    draw(ctx)
    b.render([ctx])
    b.wait()
    assert b.stats()["ctas"] == ctas
    b.destroy()
    ctx.destroy()


# ---- the sums that decide it, restated

MASK = 0xFFFFFFFF


def sat_add(a, b):
    s = (a + b) & MASK
    return MASK if s < a else s


def test_saturating_sums():
    """k_scan's sums: any grouping of saturating additions gives min(sum, 2^32 - 1), and the look-back's
    sum of 32 words in 16-bit halves does too; below the limit every sum is the plain one."""
    rng = np.random.default_rng(5)
    for case in range(300):
        hi = [10, 1 << 20, 1 << 27, 1 << 32][case % 4]
        v = [int(x) for x in rng.integers(0, hi, 64)]
        want = min(sum(v), MASK)
        left = 0
        for x in v:
            left = sat_add(left, x)
        tree = list(v)
        while len(tree) > 1:
            tree = [sat_add(tree[i], tree[i + 1]) for i in range(0, len(tree), 2)]
        assert left == tree[0] == want
        total = 0
        for g in (v[:32], v[32:]):  # two windows of the look-back
            lo = sum(x & 0xFFFF for x in g)
            h = sum(x >> 16 for x in g) + (lo >> 16)
            assert lo <= MASK and h <= MASK
            total = sat_add(total, MASK if h > 0xFFFF else (h << 16) | (lo & 0xFFFF))
        assert total == want


def test_the_pair_total_stays_past_its_capacity():
    """flush_pairs' total under any interleaving: warps add 1 to 64 pairs and take an addition back
    that found the capacity exceeded. Past the capacity it stays past it and never comes near 2^32;
    within it, it is the plain sum. (16 warps stand for the GPU's: the bound is the capacity plus 64
    for each.)"""
    rng = np.random.default_rng(6)
    for cap, adds in ((100, 5), (100, 4000), (0xF0000000, 4000), (0, 50)):
        start = max(0, cap - 20_000)  # what earlier warps added, none of it taken back
        total, plain, most = start, start, 0
        undo = []  # warps between their addition and its removal
        left = adds
        while left or undo:
            if left and len(undo) < 16 and rng.random() < 0.6:
                n = int(rng.integers(1, 65))
                left -= 1
                pos, total, plain = total, (total + n) & MASK, plain + n
                if pos > cap:
                    undo.append(n)
            elif undo:
                total = (total - undo.pop(int(rng.integers(len(undo))))) & MASK
            most = max(most, total)
            assert (total > cap) == (plain > cap)
        assert most <= cap + 64 * 17
        if plain <= cap:
            assert total == plain
