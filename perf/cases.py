"""Performance cases of the renderer: what a program that uses it has it do, pass after pass.

A pass is one frame (or one batch, or one burst of served requests) through the C ABI, from the
frame's GL calls to the finished pixels in page-locked host memory: the framebuffer lives on the
device, and a headless program takes its frames by reading them back. prepare() builds what such
a program holds before the pass: contexts with their buffer objects, textures and display lists
uploaded, the frame's encoded calls, client arrays, the batch executor or the server, and the
page-locked destinations. Sizes are those of the benchmark's workloads and the tests, or generic.
"""
import ctypes
import math

import numpy as np
import torch

import mytinygl_gb300
from mytinygl_gb300 import gl as G
from mytinygl_gb300 import workloads as W
from mytinygl_gb300.scene import Scene

RESOLUTIONS = W.SERVE_RESOLUTIONS


def listed():
    return [
        # the smallest call: an icon-sized view of a dozen triangles in immediate mode, as every
        # first GL program and every small gizmo draws them; latency and launches are all there is
        dict(name="immediate_64", kind="immediate", width=64, height=64, triangles=12, arrays="immediate"),
        # the benchmark's plain single frame: a lit sphere, colour and depth taken (RGB-D view)
        dict(name="sphere_800x600", kind="sphere", width=800, height=600, triangles=1984, texture=0, arrays="vbo"),
        # the benchmark's textured frame: clipping, eight lights, fog, trilinear texture
        dict(name="textured_1080p", kind="textured", width=1920, height=1080, triangles=100_000, texture=512,
             arrays="vbo"),
        # the benchmark's order-sensitive frame: a million small blended triangles with stencil
        dict(name="rop_1080p", kind="rop", width=1920, height=1080, triangles=1_000_000, arrays="vbo"),
        # per-fragment lighting with a specular highlight on a textured mesh, odd size
        dict(name="phong_1279x719", kind="phong", width=1279, height=719, triangles=20_000, texture=256, arrays="vbo"),
        # a wireframe editor view: mesh edges, wide axis lines and vertex points, odd size
        dict(name="wire_1021x767", kind="wire", width=1021, height=767, triangles=8_000, arrays="vbo"),
        # a particle effect in 4K: large textured quads blended over one another
        dict(name="sprites_2160p", kind="sprites", width=3840, height=2160, sprites=600, size=256, texture=128,
             arrays="client"),
        # video playback: every frame uploads a new image, draws it and blits a caption over it
        dict(name="video_720p", kind="video", width=1280, height=720, texture=1024),
        # frames whose geometry the program rewrites every time (client arrays), batched
        dict(name="batch_client_32", kind="batch", frames=32, min_side=64, max_side=1024, min_triangles=100,
             max_triangles=50_000, texture=256, arrays="client"),
        # many small views, as a simulator renders for its agents
        dict(name="batch_small_128", kind="batch", frames=128, min_side=64, max_side=160, min_triangles=100,
             max_triangles=3_000, texture=64, arrays="vbo"),
        # the benchmark's uneven batch
        dict(name="batch_uneven_256", kind="batch", frames=256, min_side=64, max_side=1024, min_triangles=100,
             max_triangles=200_000, texture=256, arrays="vbo"),
        # a burst of requests on the serving loop, over resident scenes of mixed size
        dict(name="serve_burst_48", kind="serve", requests=48, scenes=12, min_triangles=1_000,
             max_triangles=200_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["immediate", "sphere", "textured", "rop", "phong", "wire", "sprites", "video", "batch", "batch",
                       "serve"])
    if kind == "immediate":
        return dict(kind=kind, width=_log_int(rng, 16, 512), height=_log_int(rng, 16, 512),
                    triangles=_log_int(rng, 12, 3_000), arrays=rng.choice(["immediate", "list"]))
    if kind == "batch":
        frames = _log_int(rng, 2, 256)
        return dict(kind=kind, frames=frames, min_side=_log_int(rng, 16, 128), max_side=_log_int(rng, 160, 1024),
                    min_triangles=100, max_triangles=_log_int(rng, 1_000, 200_000),
                    texture=rng.choice([64, 128, 256]), arrays="client" if frames <= 32 and rng.random() < 0.5 else "vbo")
    if kind == "serve":
        return dict(kind=kind, requests=_log_int(rng, 1, 64), scenes=rng.randint(1, 16), min_triangles=1_000,
                    max_triangles=_log_int(rng, 2_000, 200_000))
    case = dict(kind=kind, width=_log_int(rng, 64, 2560), height=_log_int(rng, 64, 1600))
    if kind == "sprites":
        case["size"] = _log_int(rng, 8, 512)
        case["sprites"] = _log_int(rng, 16, max(32, min(20_000, 60_000_000 // case["size"] ** 2)))
    elif kind != "video":
        most = {"textured": 500_000, "rop": max(1_000, min(1_000_000, case["width"] * case["height"] // 2))}
        case["triangles"] = _log_int(rng, 200, most.get(kind, 100_000))
    if kind not in ("rop", "wire"):
        case["texture"] = rng.choice([64, 100, 256, 512, 1024])
    if kind != "video":
        case["arrays"] = rng.choice(["vbo", "client"])
    return case


# ---------------------------------------------------------------------------------- the frames


def _sphere_mesh(triangles):
    """A unit sphere of about `triangles` triangles: positions (its normals too), texture
    coordinates and indices."""
    n = max(3, int(round(0.5 + math.sqrt(0.25 + triangles / 2.0))))  # 2 n (n - 1) triangles
    th, ph = np.meshgrid(np.pi * np.arange(n + 1) / n, 2 * np.pi * np.arange(n + 1) / n, indexing="ij")
    pos = np.stack([np.sin(th) * np.cos(ph), np.cos(th), np.sin(th) * np.sin(ph)], -1).reshape(-1, 3).astype(np.float32)
    uv = np.stack([ph / (2 * np.pi), th / np.pi], -1).reshape(-1, 2).astype(np.float32)
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    a = i * (n + 1) + j
    b, c, d = a + n + 1, a + n + 2, a + 1
    first, second = np.stack([a, b, d], -1)[1:], np.stack([b, c, d], -1)[:-1]  # none degenerate at the poles
    idx = np.concatenate([first.reshape(-1, 3), second.reshape(-1, 3)])
    return pos, uv, np.ascontiguousarray(idx.reshape(-1).astype(np.uint32))


def _vec(*v):
    return np.array(v, np.float32)


def _upload(s, target, data, name):
    s.glBindBuffer(target, name)
    s.glBufferData(target, int(data.nbytes), data, G.GL_STATIC_DRAW)


def _texture(s, size, rng):
    s.glGenTextures(1, np.zeros(1, np.uint32))
    s.glBindTexture(G.GL_TEXTURE_2D, 1)
    s.glTexImage2D(G.GL_TEXTURE_2D, 0, G.GL_RGBA, size, size, 0, G.GL_RGBA, G.GL_UNSIGNED_BYTE,
                   rng.integers(0, 256, (size, size, 4), dtype=np.uint8))


def _camera(s, w, h, rng):
    s.glMatrixMode(G.GL_PROJECTION)
    s.glLoadIdentity()
    s.glFrustum(*W.frustum_params(60.0, w / h, 0.1, 100.0))
    s.glMatrixMode(G.GL_MODELVIEW)
    s.glLoadIdentity()
    light = rng.normal(size=3)
    light = (light / np.linalg.norm(light)).astype(np.float32)
    s.glLightfv(G.GL_LIGHT0, G.GL_POSITION, _vec(*light, 0.0))
    s.glTranslatef(0.0, 0.0, -2.5)
    s.glMultMatrixf(W.euler_matrix(*rng.uniform(0.0, 2 * math.pi, 3)))


def _mesh_frame(case, rng, style):
    """A sphere seen by a perspective camera, lit by one directional light. style: "lit" (per
    vertex, Gouraud), "phong" (per fragment, specular, linear fog) or "wire" (edges, axis lines
    and vertex points)."""
    w, h, tex = case["width"], case["height"], case.get("texture", 0)
    pos, uv, idx = _sphere_mesh(case["triangles"])
    s = Scene(style, w, h)
    if tex:
        _texture(s, tex, rng)
    vbo = case["arrays"] == "vbo"
    inter = np.ascontiguousarray(np.concatenate([pos, pos, uv], axis=1))
    if vbo:
        s.glGenBuffers(2, np.zeros(2, np.uint32))
        _upload(s, G.GL_ARRAY_BUFFER, inter, 1)
        _upload(s, G.GL_ELEMENT_ARRAY_BUFFER, idx, 2)
    s.glViewport(0, 0, w, h)
    s.glClearColor(0.0, 0.0, 0.0, 1.0)
    # ---- the frame
    s.glClear(G.GL_COLOR_BUFFER_BIT | G.GL_DEPTH_BUFFER_BIT)
    _camera(s, w, h, rng)
    s.glLightfv(G.GL_LIGHT0, G.GL_DIFFUSE, _vec(1, 1, 1, 1))
    s.glEnable(G.GL_LIGHTING)
    s.glEnable(G.GL_LIGHT0)
    s.glEnable(G.GL_DEPTH_TEST)
    s.glDepthFunc(G.GL_LESS)
    if style != "wire":
        s.glEnable(G.GL_CULL_FACE)
        s.glCullFace(G.GL_BACK)
    if style == "phong":
        s.glShadeModel(G.GL_PHONG)
        s.glLightfv(G.GL_LIGHT0, G.GL_SPECULAR, _vec(1, 1, 1, 1))
        s.glLightModeli(G.GL_LIGHT_MODEL_LOCAL_VIEWER, 1)
        s.glMaterialfv(G.GL_FRONT_AND_BACK, G.GL_SPECULAR, _vec(0.6, 0.6, 0.6, 1.0))
        s.glMaterialf(G.GL_FRONT_AND_BACK, G.GL_SHININESS, 24.0)
        s.glEnable(G.GL_FOG)
        s.glFogi(G.GL_FOG_MODE, G.GL_LINEAR)
        s.glFogf(G.GL_FOG_START, 1.0)
        s.glFogf(G.GL_FOG_END, 4.0)
        s.glFogfv(G.GL_FOG_COLOR, _vec(0.2, 0.2, 0.3, 1.0))
    if style == "wire":
        s.glPolygonMode(G.GL_FRONT_AND_BACK, G.GL_LINE)
        s.glLineWidth(1.0)
    if tex:
        s.glBindTexture(G.GL_TEXTURE_2D, 1)
        s.glTexParameteri(G.GL_TEXTURE_2D, G.GL_TEXTURE_MIN_FILTER, G.GL_LINEAR_MIPMAP_LINEAR)
        s.glTexParameteri(G.GL_TEXTURE_2D, G.GL_TEXTURE_MAG_FILTER, G.GL_LINEAR)
        s.glTexEnvi(G.GL_TEXTURE_ENV, G.GL_TEXTURE_ENV_MODE, G.GL_MODULATE)
        s.glEnable(G.GL_TEXTURE_2D)
        s.glEnableClientState(G.GL_TEXTURE_COORD_ARRAY)
    s.glEnableClientState(G.GL_VERTEX_ARRAY)
    s.glEnableClientState(G.GL_NORMAL_ARRAY)
    if vbo:
        s.glBindBuffer(G.GL_ARRAY_BUFFER, 1)
        s.glBindBuffer(G.GL_ELEMENT_ARRAY_BUFFER, 2)
        s.glVertexPointer(3, G.GL_FLOAT, 32, 0)
        s.glNormalPointer(G.GL_FLOAT, 32, 12)
        s.glTexCoordPointer(2, G.GL_FLOAT, 32, 24)
    else:
        s.glVertexPointer(3, G.GL_FLOAT, 0, pos)
        s.glNormalPointer(G.GL_FLOAT, 0, pos)
        s.glTexCoordPointer(2, G.GL_FLOAT, 0, uv)
    s.glDrawElements(G.GL_TRIANGLES, int(idx.size), G.GL_UNSIGNED_INT, 0 if vbo else idx)
    if style == "wire":
        s.glPolygonMode(G.GL_FRONT_AND_BACK, G.GL_FILL)
        s.glDisable(G.GL_LIGHTING)
        s.glColor3f(1.0, 0.8, 0.1)
        s.glPointSize(3.0)
        s.glDrawArrays(G.GL_POINTS, 0, int(pos.shape[0]))
        s.glLineWidth(3.0)
        s.glBegin(G.GL_LINES)
        for k in range(3):
            s.glColor3f(*(1.0 if i == k else 0.1 for i in range(3)))
            s.glVertex3f(0.0, 0.0, 0.0)
            s.glVertex3f(*(1.4 if i == k else 0.0 for i in range(3)))
        s.glEnd()
    return s


def _immediate_frame(case, rng):
    """Free triangles around the origin, one GL call per vertex: in immediate mode, or compiled
    into a display list beforehand."""
    w, h, n = case["width"], case["height"], case["triangles"]
    v = (rng.uniform(-1.0, 1.0, (n, 1, 3)) + rng.uniform(-0.5, 0.5, (n, 3, 3))).astype(np.float32)
    c = rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32)
    s = Scene("immediate", w, h)

    def geometry():
        s.glBegin(G.GL_TRIANGLES)
        for k in range(n):
            s.glColor3f(*(float(x) for x in c[k]))
            for p in v[k]:
                s.glVertex3f(*(float(x) for x in p))
        s.glEnd()

    if case["arrays"] == "list":
        s.glGenLists(1)
        s.glNewList(1, G.GL_COMPILE)
        geometry()
        s.glEndList()
    s.glViewport(0, 0, w, h)
    s.glClearColor(0.2, 0.2, 0.2, 1.0)
    # ---- the frame
    s.glClear(G.GL_COLOR_BUFFER_BIT | G.GL_DEPTH_BUFFER_BIT)
    _camera(s, w, h, rng)
    s.glEnable(G.GL_DEPTH_TEST)
    s.glDepthFunc(G.GL_LESS)
    if case["arrays"] == "list":
        s.glCallList(1)
    else:
        geometry()
    return s


def _sprites_frame(case, rng):
    """Square textured quads of `size` pixels anywhere on the screen, blended back to front."""
    w, h, n, size = case["width"], case["height"], case["sprites"], case["size"]
    centre = rng.uniform(-1.0, 1.0, (n, 1, 2))
    corner = np.array([[-1, -1], [1, -1], [1, 1], [-1, 1]], np.float64) * [size / w, size / h]
    z = np.broadcast_to(np.linspace(0.9, -0.9, n)[:, None, None], (n, 4, 1))
    pos = np.ascontiguousarray(np.concatenate([centre + corner, z], axis=2).reshape(-1, 3).astype(np.float32))
    uv = np.ascontiguousarray(np.tile(_vec(0, 0, 1, 0, 1, 1, 0, 1), n).reshape(-1, 2))
    col = np.ascontiguousarray(np.repeat(rng.integers(0, 256, (n, 4), dtype=np.uint8), 4, axis=0))
    s = Scene("sprites", w, h)
    _texture(s, case["texture"], rng)
    vbo = case["arrays"] == "vbo"
    if vbo:  # one interleaved buffer: position f32x3 | uv f32x2 | colour u8x4
        rec = np.zeros(4 * n, dtype=[("p", "<f4", 3), ("t", "<f4", 2), ("c", "u1", 4)])
        rec["p"], rec["t"], rec["c"] = pos, uv, col
        s.glGenBuffers(1, np.zeros(1, np.uint32))
        _upload(s, G.GL_ARRAY_BUFFER, np.frombuffer(rec.tobytes(), np.uint8), 1)
    s.glViewport(0, 0, w, h)
    s.glClearColor(0.05, 0.05, 0.1, 1.0)
    # ---- the frame
    s.glClear(G.GL_COLOR_BUFFER_BIT)
    for m in (G.GL_PROJECTION, G.GL_MODELVIEW):
        s.glMatrixMode(m)
        s.glLoadIdentity()
    s.glBindTexture(G.GL_TEXTURE_2D, 1)
    s.glTexParameteri(G.GL_TEXTURE_2D, G.GL_TEXTURE_MIN_FILTER, G.GL_LINEAR)
    s.glTexParameteri(G.GL_TEXTURE_2D, G.GL_TEXTURE_MAG_FILTER, G.GL_LINEAR)
    s.glTexEnvi(G.GL_TEXTURE_ENV, G.GL_TEXTURE_ENV_MODE, G.GL_MODULATE)
    s.glEnable(G.GL_TEXTURE_2D)
    s.glEnable(G.GL_ALPHA_TEST)
    s.glAlphaFunc(G.GL_GREATER, 0.05)
    s.glEnable(G.GL_BLEND)
    s.glBlendFunc(G.GL_SRC_ALPHA, G.GL_ONE_MINUS_SRC_ALPHA)
    for a in (G.GL_VERTEX_ARRAY, G.GL_COLOR_ARRAY, G.GL_TEXTURE_COORD_ARRAY):
        s.glEnableClientState(a)
    stride = 24 if vbo else 0
    s.glVertexPointer(3, G.GL_FLOAT, stride, 0 if vbo else pos)
    s.glTexCoordPointer(2, G.GL_FLOAT, stride, 12 if vbo else uv)
    s.glColorPointer(4, G.GL_UNSIGNED_BYTE, stride, 20 if vbo else col)
    s.glDrawArrays(G.GL_QUADS, 0, 4 * n)
    return s


def _video_frame(case, rng):
    """A full-screen quad of an image uploaded for this frame, and a caption blitted over it."""
    w, h, size = case["width"], case["height"], case["texture"]
    s = Scene("video", w, h)
    s.glGenTextures(1, np.zeros(1, np.uint32))
    s.glViewport(0, 0, w, h)
    # ---- the frame
    s.glClear(G.GL_COLOR_BUFFER_BIT)
    s.glBindTexture(G.GL_TEXTURE_2D, 1)
    s.glTexImage2D(G.GL_TEXTURE_2D, 0, G.GL_RGBA, size, size, 0, G.GL_RGBA, G.GL_UNSIGNED_BYTE,
                   rng.integers(0, 256, (size, size, 4), dtype=np.uint8))
    s.glTexParameteri(G.GL_TEXTURE_2D, G.GL_TEXTURE_MIN_FILTER, G.GL_LINEAR)
    s.glTexParameteri(G.GL_TEXTURE_2D, G.GL_TEXTURE_MAG_FILTER, G.GL_LINEAR)
    s.glTexEnvi(G.GL_TEXTURE_ENV, G.GL_TEXTURE_ENV_MODE, G.GL_REPLACE)
    s.glEnable(G.GL_TEXTURE_2D)
    s.glBegin(G.GL_QUADS)
    for x, y in ((0, 0), (1, 0), (1, 1), (0, 1)):
        s.glTexCoord2f(float(x), float(y))
        s.glVertex2f(2.0 * x - 1.0, 2.0 * y - 1.0)
    s.glEnd()
    s.glDisable(G.GL_TEXTURE_2D)
    cw, ch = max(1, w // 2), max(1, h // 12)
    s.glRasterPos2f(-0.5, -0.9)
    s.glDrawPixels(cw, ch, G.GL_RGBA, G.GL_UNSIGNED_BYTE, rng.integers(0, 256, (ch, cw, 4), dtype=np.uint8))
    return s


def _scene(case, rng):
    kind = case["kind"]
    if kind in ("textured", "rop"):
        kw = dict(tex_size=case["texture"]) if kind == "textured" else {}
        return W.HEADLINE[kind](case["width"], case["height"], ntri=case["triangles"], seed=int(rng.integers(1 << 31)),
                                use_vbo=case["arrays"] == "vbo", **kw)
    if kind == "immediate":
        return _immediate_frame(case, rng)
    if kind == "sprites":
        return _sprites_frame(case, rng)
    if kind == "video":
        return _video_frame(case, rng)
    return _mesh_frame(case, rng, {"sphere": "lit"}.get(kind, kind))


def _batch_plan(case):
    """The frames of a batch: each a single-frame case of its own size (fixed by the case)."""
    rng = np.random.default_rng([9, case["frames"], case["max_side"], case["max_triangles"]])

    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    return [dict(kind=("sphere", "textured")[int(rng.integers(2))], width=log(case["min_side"], case["max_side"]),
                 height=log(case["min_side"], case["max_side"]),
                 triangles=log(case["min_triangles"], case["max_triangles"]), texture=case["texture"],
                 arrays=case["arrays"]) for _ in range(case["frames"])]


def _serve_plan(case):
    """Triangles and texture of each resident scene; scene and resolution of each request."""
    rng = np.random.default_rng([10, case["requests"], case["scenes"], case["max_triangles"]])
    lo, hi = math.log(case["min_triangles"]), math.log(case["max_triangles"])
    scenes = [(int(round(math.exp(rng.uniform(lo, hi)))), int(2 ** rng.integers(8, 11))) for _ in range(case["scenes"])]
    return scenes, [(int(rng.integers(len(scenes))), RESOLUTIONS[int(rng.integers(len(RESOLUTIONS)))])
                    for _ in range(case["requests"])]


# ---------------------------------------------------------------------------------- measured interface


def _pinned(*shape, dtype=torch.uint8):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def _flat_frames(sizes):
    """One page-locked buffer for all frames and each frame's address in it (64-byte steps)."""
    starts, at = [], 0
    for w, h in sizes:
        starts.append(at)
        at += (4 * w * h + 63) // 64 * 64
    flat = _pinned(at)
    flat.zero_()
    return flat, [flat.data_ptr() + a for a in starts]


def _resident(lib, scene):
    """A context with the scene's resident part uploaded, and the stream of its frame."""
    ctx = lib.context(scene.width, scene.height)
    k = W.frame_start(scene)
    scene.play(ctx, 0, k)
    ctx.finish()
    return ctx, scene.stream(k)


def prepare(case, seed):
    lib = mytinygl_gb300.library()
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "batch":
        plan = _batch_plan(case)
        scenes = [_scene(c, rng) for c in plan]
        pairs = [_resident(lib, s) for s in scenes]
        ctxs = [c for c, _ in pairs]
        flat, dst = _flat_frames([(c["width"], c["height"]) for c in plan])
        n = len(ctxs)
        return dict(kind=kind, batch=lib.batch(), streams=G.PreparedStreams(lib, ctxs, [s for _, s in pairs]),
                    handles=(ctypes.c_void_p * n)(*[c.handle for c in ctxs]), dst=(ctypes.c_void_p * n)(*dst), n=n,
                    lib=lib, out=flat, contexts=ctxs, scenes=scenes)
    if kind == "serve":
        plan, requests = _serve_plan(case)
        scenes = [W.textured_scene(1920, 1080, ntri=n, seed=int(rng.integers(1 << 31)), tex_size=t,
                                   modelview_from_caller=True) for n, t in plan]
        server = lib.server()
        ctxs = []
        for s in scenes:
            ctx, stream = _resident(lib, s)
            server.add_scene(ctx, stream, W.scene_triangles(s))
            ctxs.append(ctx)
        flat, dst = _flat_frames([r for _, r in requests])
        reqs = (G.Request * len(requests))()
        for q, (sc, (w, h)), d in zip(reqs, requests, dst):
            q.scene, q.width, q.height, q.color, q.arrival = sc, w, h, d, 0.0
            q.modelview[:] = W.euler_matrix(rng.uniform(-0.3, 0.3), rng.uniform(-0.3, 0.3), rng.uniform(0, 2 * math.pi))
        return dict(kind=kind, server=server, reqs=reqs, out=flat, contexts=ctxs, scenes=scenes)
    scene = _scene(case, rng)
    ctx, stream = _resident(lib, scene)
    w, h = scene.width, scene.height
    out = [_pinned(h, w, 4),
           _pinned(h, w, dtype=torch.float32) if kind in ("sphere", "textured", "wire") else None,
           _pinned(h, w) if kind == "rop" else None]
    return dict(kind=kind, streams=G.PreparedStreams(lib, [ctx], [stream]), handle=ctx.handle,
                dst=[t.data_ptr() if t is not None else None for t in out], lib=lib,
                out=[t for t in out if t is not None], contexts=[ctx], scenes=[scene])


def run(state):
    kind = state["kind"]
    if kind == "serve":
        state["server"].run_trace(state["reqs"])
        return state["out"]
    state["streams"].play()
    if kind == "batch":
        batch = state["batch"]
        st = state["lib"].lib.mtgl_batch_render_read(batch.handle, state["handles"], state["dst"], state["n"])
        if st != 0:
            raise RuntimeError(f"mtgl_batch_render_read failed with status {st}")
        batch.wait()
        return state["out"]
    st = state["lib"].lib.mtgl_read_framebuffer(state["handle"], *state["dst"])
    if st != 0:
        raise RuntimeError(f"mtgl_read_framebuffer failed with status {st}")
    return state["out"]


def exact(case, seed):
    """None: the colours and stencils are bytes, and which fragment a pixel keeps (so its depth
    too) is decided by 32-bit coverage and depth comparisons whose rounding is the result."""
    return None


def work(case):
    """Bytes: vertex attributes, indices and textures read once, the returned buffers written
    once. Operations: the transforms and lighting of every vertex, and one shading of every
    pixel (of every fragment where they blend)."""
    kind = case["kind"]
    if kind == "batch":
        parts = [work(c) for c in _batch_plan(case)]
        depth = sum(4.0 * c["width"] * c["height"] for c in _batch_plan(case))  # colour alone is returned
        return {"bytes": sum(p["bytes"] for p in parts) - depth, "flops": sum(p["flops"] for p in parts)}
    if kind == "serve":
        scenes, requests = _serve_plan(case)
        total = {"bytes": 0.0, "flops": 0.0}
        for k, (w, h) in requests:
            p = work(dict(kind="textured", width=w, height=h, triangles=scenes[k][0], texture=scenes[k][1]))
            total["bytes"] += p["bytes"] - 4.0 * w * h
            total["flops"] += p["flops"]
        return total
    pixels = case["width"] * case["height"]
    tri, tex = case.get("triangles", 2), case.get("texture", 0)
    if kind in ("sphere", "phong", "wire"):  # an indexed mesh: about half as many vertices as triangles
        verts, vbytes, lights, frags = tri // 2, 32, 1, pixels // 3
    elif kind == "textured":
        verts, vbytes, lights, frags = 3 * tri, 36, 8, pixels
    elif kind == "rop":
        verts, vbytes, lights, frags = 3 * tri, 16, 0, 33 * tri  # mean of the log-normal areas
    elif kind == "sprites":
        verts, vbytes, lights, frags = 4 * case["sprites"], 24, 0, case["sprites"] * case["size"] ** 2
    elif kind == "video":
        verts, vbytes, lights, frags = 4, 24, 0, pixels
    else:
        verts, vbytes, lights, frags = 3 * tri, 24, 0, pixels // 3
    indices = 12 * tri if kind in ("sphere", "phong", "wire") else 0
    out = pixels * (4 + (4 if kind in ("sphere", "textured", "wire") else 0) + (1 if kind == "rop" else 0))
    return {"bytes": float(verts * vbytes + indices + 4 * tex * tex + out),
            "flops": float(verts * (150 + 45 * lights) + frags * (200 if kind == "phong" else 60))}
