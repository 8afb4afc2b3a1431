"""Renders one benchmark workload's frame a few times in a row, for profilers.

    python -m mytinygl_gb300.profile_frame --workload textured --frames 3
    python -m mytinygl_gb300.profile_frame --workload batch --frames 3 [--batch-frames 256]
    python -m mytinygl_gb300.profile_frame --workload block-fog

Each frame is the workload's per-frame GL calls followed by glFinish, on one context, with
nothing else on the GPU in between (no cache flush, no timing events), so a profiler's
capture of the n-th frame's kernels sees what the previous frame left in L2 and nothing
else. `batch` renders the uneven batch of bench.py (256 contexts, one mtgl_batch_render per
repetition, the batch's defaults). Workloads are those of mytinygl_gb300/workloads.py.
`block-*` are 1920x1080 frames of one triangle, for what a tile costs by itself: empty (it
covers two dozen pixels), flat, bilinear (512^2 texture), fog (the same with linear fog). Their
frames are read back into page-locked memory, so the tile launch writes that too.
"""
from __future__ import annotations

import argparse
import ctypes

import numpy as np

from . import gl as G
from . import library
from . import workloads as W
from .scene import Scene


def block_scene(stages):
    s = Scene("block", 1920, 1080)
    if stages in ("bilinear", "fog"):
        s.glGenTextures(1, np.zeros(1, np.uint32))
        s.glBindTexture(G.GL_TEXTURE_2D, 1)
        s.glTexImage2D(G.GL_TEXTURE_2D, 0, G.GL_RGBA, 512, 512, 0, G.GL_RGBA, G.GL_UNSIGNED_BYTE,
                       np.random.default_rng(1).integers(0, 256, (512, 512, 4), dtype=np.uint8))
    s.glViewport(0, 0, 1920, 1080)
    s.glClearColor(0.0, 0.0, 0.0, 1.0)
    s.glClear(G.GL_COLOR_BUFFER_BIT | G.GL_DEPTH_BUFFER_BIT)
    s.glEnable(G.GL_DEPTH_TEST)
    s.glDepthFunc(G.GL_LESS)
    if stages in ("bilinear", "fog"):
        s.glTexParameteri(G.GL_TEXTURE_2D, G.GL_TEXTURE_MIN_FILTER, G.GL_LINEAR)
        s.glTexParameteri(G.GL_TEXTURE_2D, G.GL_TEXTURE_MAG_FILTER, G.GL_LINEAR)
        s.glEnable(G.GL_TEXTURE_2D)
    if stages == "fog":
        s.glEnable(G.GL_FOG)
        s.glFogi(G.GL_FOG_MODE, G.GL_LINEAR)
        s.glFogf(G.GL_FOG_START, 1.0)
        s.glFogf(G.GL_FOG_END, 4.0)
    size, at = (0.01, 0.0) if stages == "empty" else (3.0, 1.0)
    s.glBegin(G.GL_TRIANGLES)
    for x, y in ((-1, -1), (1, -1), (-1, 1)):
        s.glTexCoord2f(x * 1.7, y * 1.9)
        s.glVertex3f(size * x + at, size * y + at, 0.9)
    s.glEnd()
    return s


SCENES = {
    "textured": W.textured_scene,
    "rop": W.rop_scene,
    "sphere": W.sphere_scene,
}
SCENES.update({f"block-{k}": (lambda k=k: block_scene(k)) for k in ("empty", "flat", "bilinear", "fog")})


def main():
    ap = argparse.ArgumentParser(description=__doc__, formatter_class=argparse.RawDescriptionHelpFormatter)
    ap.add_argument("--workload", choices=sorted(SCENES) + ["batch"], default="textured")
    ap.add_argument("--frames", type=int, default=3, help="repetitions")
    ap.add_argument("--batch-frames", type=int, default=256)
    args = ap.parse_args()
    lib = library()
    if args.workload == "batch":
        scenes = W.uneven_batch(args.batch_frames)
        ctxs, streams = [], []
        for sc in scenes:
            c = lib.context(sc.width, sc.height)
            k = W.frame_start(sc)
            sc.play(c, 0, k)
            c.glFinish()
            ctxs.append(c)
            streams.append(sc.stream(k))
        b = lib.batch()
        for _ in range(args.frames):
            lib.play_many(ctxs, streams)
            b.render(ctxs)
            b.wait()
        print(f"batch of {len(scenes)}: {args.frames} runs, stats {b.stats()}")
        b.destroy()
        for c in ctxs:
            c.destroy()
        return
    scene = SCENES[args.workload]()
    fs = W.frame_start(scene)
    ctx = lib.context(scene.width, scene.height)
    scene.play(ctx, 0, fs)
    ctx.glFinish()
    host = None
    if args.workload.startswith("block-"):
        import torch

        host = torch.empty((scene.height, scene.width, 4), dtype=torch.uint8, pin_memory=True)
    for _ in range(args.frames):
        scene.play(ctx, fs)
        if host is None:
            ctx.glFinish()
        elif lib.lib.mtgl_read_framebuffer(ctx.handle, ctypes.c_void_p(host.data_ptr()), None, None):
            raise RuntimeError("read-back failed")
    print(f"{args.workload}: {args.frames} frames, stats {ctx.stats()}")
    ctx.destroy()


if __name__ == "__main__":
    main()
