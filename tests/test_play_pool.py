"""mtgl_play_many's helper threads, kept between calls: several callers at once, after an idle
spell, and in a forked child, against the same streams played one by one (CPU back end)."""
import importlib
import os
import subprocess
import sys
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


STUBS = r"""
#include "fe_internal.h"
#include <unistd.h>
int mtgl_dev_in_batch(const mtgl_dev *d) { (void)d; return 0; }
GLState *gl_get_current_context(void) { return NULL; }
void gl_make_current(GLState *c) { (void)c; }
int mtgl_play(GLState *c, const void *s, size_t n) { (void)c; (void)s; (void)n; usleep(20000); return 0; }
"""
SLOW = r"""
#define _GNU_SOURCE
#include <pthread.h>
#include <unistd.h>
int slow_unlock(pthread_mutex_t *m)  /* the other threads are slow to return from it */
{
    const int r = pthread_mutex_unlock(m);
    if (gettid() != getpid()) usleep(200000);
    return r;
}
"""
UNLOAD = r"""
import _ctypes, ctypes, sys, time
ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)
for _ in range(2):
    lib = ctypes.CDLL(sys.argv[2])
    states = [ctypes.create_string_buffer(1 << 20) for _ in range(8)]
    ctxs = (ctypes.c_void_p * 8)(*[ctypes.addressof(b) for b in states])
    assert lib.mtgl_play_many(ctxs, (ctypes.c_void_p * 8)(), (ctypes.c_size_t * 8)(), 8) == 0
    _ctypes.dlclose(lib._handle)
    assert sys.argv[2] not in open("/proc/self/maps").read()
    time.sleep(0.6)
"""


def test_unloading_waits_for_the_helpers_to_leave(tmp_path):
    """The library is unloaded right after a call: no helper may still be on its way out of its code,
    however slowly it returns from its last unlock."""
    B = importlib.import_module("mytinygl_gb300.build")
    (tmp_path / "stubs.c").write_text(STUBS)
    (tmp_path / "slow.c").write_text(SLOW)
    slow, play = str(tmp_path / "libslow.so"), str(tmp_path / "libplay.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-pthread", "-o", slow, str(tmp_path / "slow.c")], check=True)
    subprocess.run(["gcc"] + B.CC_FLAGS + [f"-I{B.FRONT_DIR}", "-pthread", "-Dpthread_mutex_unlock=slow_unlock", "-shared",
                    "-o", play, os.path.join(B.FRONT_DIR, "fe_play_many.c"), str(tmp_path / "stubs.c"), slow], check=True)
    r = subprocess.run([sys.executable, "-c", UNLOAD, slow, play], env=dict(os.environ, MTGL_PLAY_THREADS="4"),
                       capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
