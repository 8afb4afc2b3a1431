"""mtgl_play_many's helper threads, kept between calls: several callers at once, after an idle
spell, and in a forked child, against the same streams played one by one (CPU back end)."""
import os
import threading
import time

import numpy as np

import harness
from mytinygl_gb300 import gl as G
from mytinygl_gb300 import workloads as W


def group(lib, seed, n=24):
    scenes = [W.sphere_scene(40 + 3 * i, 33, seed=seed + i, stacks=5, slices=6, use_vbo=bool(i % 2)) for i in range(n)]
    ctxs = [lib.context(s.width, s.height) for s in scenes]
    for c, s in zip(ctxs, scenes):
        s.play(c, 0, W.frame_start(s))
    return scenes, ctxs, G.PreparedStreams(lib, ctxs, [s.stream(W.frame_start(s)) for s in scenes])


def frames(ctxs):
    return [c.read() for c in ctxs]


def same(a, b):
    return all(np.array_equal(x, y) for f, g in zip(a, b) for x, y in zip(f, g))


def test_concurrent_callers_idle_helpers_and_a_fork():
    lib = harness.oracle()
    os.environ["MTGL_PLAY_THREADS"] = "6"
    try:
        groups = [group(lib, 100 * k) for k in range(3)]
        want = []
        for scenes, _, _ in groups:
            want.append([])
            for s in scenes:
                c = lib.context(s.width, s.height)
                s.play(c)
                want[-1].append(c.read())
                c.destroy()
        failed = []

        def caller(k):
            try:
                for _ in range(20):
                    groups[k][2].play()
                if not same(frames(groups[k][1]), want[k]):
                    failed.append(k)
            except Exception as e:  # reported below: threads swallow it
                failed.append((k, repr(e)))

        threads = [threading.Thread(target=caller, args=(k,)) for k in range(3)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not failed
        time.sleep(2.3)  # the helpers end
        groups[0][2].play()
        assert same(frames(groups[0][1]), want[0])
        pid = os.fork()
        if pid == 0:  # no helper lives here; new ones start
            ok = False
            try:
                groups[1][2].play()
                ok = same(frames(groups[1][1]), want[1])
            finally:
                os._exit(0 if ok else 1)
        assert os.waitpid(pid, 0)[1] == 0
        for _, ctxs, _ in groups:
            for c in ctxs:
                c.destroy()
    finally:
        os.environ.pop("MTGL_PLAY_THREADS", None)
