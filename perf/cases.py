"""Measured cases: the flushes a program has the backend do.

A case is one frame, or one batch of frames, from its flush records to the
finished RGBA8 target(s), through the C ABI (include/rive_cuda.h) and its
Python binding. The scenes are this repository's own distributions (scene.py:
plain fills, full-feature paths, stroke stress), generic user-interface
screens, and the recorded frames under tests/golden with every path moved and
every colour and image changed by the seed. Records of synthetic scenes come
from the front-end stand-in that `__graft_entry__.build()` compiles.
"""
import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package (its directory's name is no identifier)."""
    if "rive_runtime_gb300" not in sys.modules:
        root = os.path.join(REPO, "rive-runtime_gb300")
        spec = importlib.util.spec_from_file_location(
            "rive_runtime_gb300", os.path.join(root, "__init__.py"),
            submodule_search_locations=[root])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["rive_runtime_gb300"] = mod
        spec.loader.exec_module(mod)
    from rive_runtime_gb300 import capture, rive_cuda, scene
    return capture, rive_cuda, scene


# Recorded frames by what they draw. `mix` frames use every draw type: feathers
# below and through the atlas, image paints, an image mesh, clips, triangulated
# fills.
RECORDED = {
    "feathered": ["silver_police_files_f60"],
    "images": ["silver_superbowl_images_f5"],
    "mix": ["silver_artboards_opacity_f30", "silver_bankcard_f10", "silver_clipping_images_f6",
            "silver_data_viz_f6", "silver_echo_show_f0", "silver_hunter_x_f0",
            "silver_image_mesh_f10", "silver_path_effect_feathers_f30", "silver_path_opacity_f30",
            "silver_police_files_f60", "silver_rewards_atlas_f10", "silver_rewards_f10",
            "silver_spotify_kids_f31", "silver_superbowl_images_f5",
            "silver_text_feather_falloff_f30", "tri_full_s23"],
}


def listed():
    return [
        # A widget redrawn alone: a handful of shapes, all launch latency.
        {"name": "ui_widget_240x180", "scene": "ui", "call": "device", "frames": 1,
         "width": 240, "height": 180, "paths": 9},
        # The same size for a render thread that may not allocate.
        {"name": "noalloc_fills_320x256", "scene": "plain", "call": "noalloc", "frames": 1,
         "width": 320, "height": 256, "paths": 30},
        # The plain small workload: 200 fills of 8 cubics on 512x512.
        {"name": "plain_fills_512", "scene": "plain", "call": "device", "frames": 1,
         "width": 512, "height": 512, "paths": 200},
        # An application's frame: records uploaded, flushed, read back.
        {"name": "app_ui_1080x1920", "scene": "ui", "call": "app", "frames": 1,
         "width": 1080, "height": 1920, "paths": 140},
        # A recorded frame with feathered fills and strokes.
        {"name": "recorded_feathered_1080", "scene": "feathered", "call": "device", "frames": 1},
        # Recorded frames of different applications served as one batch.
        {"name": "recorded_mix_batch", "scene": "mix", "call": "batch", "frames": 16},
        # Screens of many sessions served as one batch, and replayed as a graph.
        {"name": "ui_batch_64", "scene": "ui", "call": "batch", "frames": 64,
         "width": 800, "height": 600, "paths": 60},
        {"name": "ui_graph_48", "scene": "ui", "call": "graph", "frames": 48,
         "width": 701, "height": 913, "paths": 45},
        # Full-feature paths (strokes, gradients, blend modes, nested clips) on
        # an odd canvas, and at full size with the work-queue raster the
        # autotuner takes for it.
        {"name": "full_feature_1021x767", "scene": "full", "call": "device", "frames": 1,
         "width": 1021, "height": 767, "paths": 900},
        {"name": "full_feature_2048", "scene": "full", "call": "device", "frames": 1,
         "width": 2048, "height": 2048, "paths": 5000, "queue": True},
        # Tessellation-heavy strokes with cusps.
        {"name": "strokes_1024", "scene": "strokes", "call": "device", "frames": 1,
         "width": 1024, "height": 1024, "paths": 5000},
        # Plain canvases of uneven size and path count in one batch.
        {"name": "plain_batch_20", "scene": "plain", "call": "batch", "frames": 20,
         "width": 760, "height": 680, "paths": 400},
    ]


def draw(rng):
    def logu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    scene = rng.choice(["ui", "ui", "plain", "full", "strokes", "feathered", "images", "mix"])
    if scene in ("feathered", "images", "mix"):
        most = {"feathered": 12, "images": 12, "mix": 16}[scene]
        return {"scene": scene, "frames": logu(1, most), "call": rng.choice(["device", "batch", "graph"]),
                "shift": logu(2, 60)}
    c = {"scene": scene, "width": logu(160, 2048), "height": logu(160, 2048)}
    if scene == "ui":
        c["paths"] = logu(5, 240)
        c["call"] = rng.choice(["device", "app", "batch", "graph"])
        c["frames"] = logu(2, 64) if c["call"] in ("batch", "graph") else 1
    elif scene == "plain":
        c["paths"] = logu(20, 800)
        c["call"] = rng.choice(["device", "app", "batch", "graph"])
        c["frames"] = logu(2, 10) if c["call"] in ("batch", "graph") else 1
    else:
        # The path density of the full-size scenes.
        area = c["width"] * c["height"] / 2048.0 ** 2
        c["paths"] = max(20, int(5000 * area * rng.uniform(0.3, 1.0)))
        c["call"] = rng.choice(["device", "app"])
        c["frames"] = 1
        if scene == "full" and rng.random() < 0.5:
            c["queue"] = True
    return c


# ---- scenes -----------------------------------------------------------------


def _rounded_rect(S, x, y, w, h, r):
    """A rounded rectangle with cubic corners, clockwise."""
    k = 0.5523 * r
    pts = [(x + r, y), (x + w - r, y), (x + w - r + k, y), (x + w, y + r - k), (x + w, y + r),
           (x + w, y + h - r), (x + w, y + h - r + k), (x + w - r + k, y + h), (x + w - r, y + h),
           (x + r, y + h), (x + r - k, y + h), (x, y + h - r + k), (x, y + h - r),
           (x, y + r), (x, y + r - k), (x + r - k, y), (x + r, y)]
    verbs = [S.VERB_MOVE] + [S.VERB_LINE, S.VERB_CUBIC] * 4 + [S.VERB_CLOSE]
    return verbs, pts


def _ellipse(S, cx, cy, rx, ry):
    kx, ky = 0.5523 * rx, 0.5523 * ry
    pts = [(cx + rx, cy), (cx + rx, cy + ky), (cx + kx, cy + ry), (cx, cy + ry),
           (cx - kx, cy + ry), (cx - rx, cy + ky), (cx - rx, cy), (cx - rx, cy - ky),
           (cx - kx, cy - ry), (cx, cy - ry), (cx + kx, cy - ry), (cx + rx, cy - ky), (cx + rx, cy)]
    return [S.VERB_MOVE] + [S.VERB_CUBIC] * 4 + [S.VERB_CLOSE], pts


def _glyphs(S, rng, x, y, size, count):
    """A line of text: per glyph an outline of lines and cubics about its cell
    and, for some, a counter of the other winding."""
    verbs, pts = [], []
    for g in range(count):
        cx, cy = x + (g + .5) * size * .62, y
        for hole in range(1 + int(rng.random() < .4)):
            n = int(rng.integers(4, 9))
            r = size * (.42 if not hole else .18)
            a = np.linspace(0, 2 * math.pi, n, endpoint=False) * (-1 if hole else 1)
            rad = r * rng.uniform(.7, 1.1, n)
            px, py = cx + .8 * rad * np.cos(a), cy + rad * np.sin(a)
            verbs.append(S.VERB_MOVE)
            pts.append((px[0], py[0]))
            for i in range(1, n + 1):
                j = i % n
                if rng.random() < .5:
                    verbs.append(S.VERB_LINE)
                else:
                    d = rng.uniform(-.15, .15, 4) * size
                    pts.append((px[i - 1] + d[0], py[i - 1] + d[1]))
                    pts.append((px[j] + d[2], py[j] + d[3]))
                    verbs.append(S.VERB_CUBIC)
                pts.append((px[j], py[j]))
            verbs.append(S.VERB_CLOSE)
    return verbs, pts


def _gradient(S, rng, paint, x, y, w, h):
    n = int(rng.integers(2, 5))
    paint.stops = [(float(p), int(rng.integers(0, 1 << 24)) | 0xFF000000)
                   for p in np.linspace(0, 1, n)]
    if rng.random() < .6:
        paint.shader = S.SHADER_LINEAR
        paint.g = (x, y, x + w * float(rng.integers(0, 2)), y + h)
    else:
        paint.shader = S.SHADER_RADIAL
        paint.g = (x + w / 2, y + h / 2, max(w, h) * .7, 0.0)


def ui_scene(S, rng, width, height, paths):
    """A screen: a backdrop, cards (rounded rectangles, gradients, borders),
    icons, lines of text and charts, some under a rounded clip."""
    sc = S.Scene(width, height, clear_color=0xFFFFFFFF)

    def put(verbs, pts, paint, rule=S.FILL_NONZERO):
        sc.cmd(S.CMD_DRAW_PATH, sc.add_path(S.Path(verbs, np.array(pts, np.float32), rule)),
               sc.add_paint(paint))

    def colour(alpha=None):
        a = 255 if alpha is None else int(alpha)
        return (a << 24) | int(rng.integers(0, 1 << 24))

    back = S.Paint(color=colour())
    _gradient(S, rng, back, 0.0, 0.0, float(width), float(height))
    put([S.VERB_MOVE, S.VERB_LINE, S.VERB_LINE, S.VERB_LINE, S.VERB_CLOSE],
        [(0, 0), (width, 0), (width, height), (0, height)], back)
    unit = math.sqrt(width * height / max(paths, 4))
    while len(sc.paths) < paths:
        x, y = rng.uniform(-.05, .9) * width, rng.uniform(-.05, .9) * height
        w, h = unit * rng.uniform(.8, 3.), unit * rng.uniform(.5, 1.6)
        kind = rng.random()
        if kind < .35:  # a card, some with a border
            clipped = rng.random() < .2
            sc.cmd(S.CMD_SAVE)
            if clipped:
                v, p = _rounded_rect(S, x + w * .1, y + h * .1, w * .9, h, min(w, h) * .2)
                sc.cmd(S.CMD_CLIP_PATH, sc.add_path(S.Path(v, np.array(p, np.float32))))
            v, p = _rounded_rect(S, x, y, w, h, min(w, h) * rng.uniform(.08, .4))
            paint = S.Paint(color=colour(rng.integers(120, 256)))
            if rng.random() < .5:
                _gradient(S, rng, paint, x, y, w, h)
            if rng.random() < .08:
                paint.blend_mode = int(S.BLEND_MODES[int(rng.integers(0, 16))])
            put(v, p, paint)
            if rng.random() < .5:
                put(v, p, S.Paint(style=S.STYLE_STROKE, color=colour(), join=S.JOIN_ROUND,
                                  thickness=float(rng.uniform(1, 4))))
            sc.cmd(S.CMD_RESTORE)
        elif kind < .55:  # an icon
            v, p = _ellipse(S, x, y, unit * .3, unit * .3 * rng.uniform(.6, 1.2))
            v2, p2 = _ellipse(S, x, y, unit * .14, unit * .14)
            put(v + v2, p + p2, S.Paint(color=colour(rng.integers(160, 256))), S.FILL_EVENODD)
        elif kind < .85:  # a line of text
            size = float(np.clip(unit * rng.uniform(.12, .4), 9, 48))
            v, p = _glyphs(S, rng, x, y, size, int(rng.integers(3, 24)))
            put(v, p, S.Paint(color=colour()))
        else:  # a chart line
            n = int(rng.integers(4, 20))
            px = np.linspace(x, x + 2 * w, n)
            py = y + h * rng.random(n)
            verbs, pts = [S.VERB_MOVE], [(px[0], py[0])]
            for i in range(1, n):
                mx = (px[i - 1] + px[i]) / 2
                pts += [(mx, py[i - 1]), (mx, py[i]), (px[i], py[i])]
                verbs.append(S.VERB_CUBIC)
            put(verbs, pts, S.Paint(style=S.STYLE_STROKE, color=colour(),
                                    join=int(rng.integers(0, 3)), cap=int(rng.integers(0, 3)),
                                    thickness=float(rng.uniform(1, 8))))
    return sc


def _planner():
    lib = ctypes.CDLL(os.path.join(REPO, "tests", "inputgen", "_build", "librive_planner.so"))
    lib.rive_plan_scene.restype = ctypes.c_int
    lib.rive_plan_scene.argtypes = [ctypes.c_void_p, ctypes.c_size_t,
                                    ctypes.POINTER(ctypes.c_void_p), ctypes.POINTER(ctypes.c_size_t),
                                    ctypes.c_char_p, ctypes.c_size_t]
    lib.rive_plan_free.restype = None
    lib.rive_plan_free.argtypes = [ctypes.c_void_p]
    return lib


def _plan(lib, capture, data):
    out, n, err = ctypes.c_void_p(), ctypes.c_size_t(), ctypes.create_string_buffer(512)
    rc = lib.rive_plan_scene(data, len(data), ctypes.byref(out), ctypes.byref(n), err, 512)
    if rc:
        raise RuntimeError("the front end failed (%d): %s" % (rc, err.value.decode()))
    try:
        return capture.parse(ctypes.string_at(out, n.value))
    finally:
        lib.rive_plan_free(out)


def _recorded(capture, name, rng, shift):
    """A recorded frame, every path moved by up to `shift` pixels and every
    solid colour and image texel changed."""
    with open(os.path.join(REPO, "tests", "golden", name + ".cap"), "rb") as f:
        cap = capture.parse(f.read())
    paths = np.frombuffer(cap.buffers["paths"], np.float32).reshape(-1, 16).copy()
    paths[1:, 4:6] += rng.uniform(-shift, shift, (len(paths) - 1, 2)).astype(np.float32)
    cap.buffers["paths"] = paths.tobytes()
    paints = np.frombuffer(cap.buffers["paints"], np.uint32).reshape(-1, 2).copy()
    solid = (paints[:, 0] & 0xF) == 1
    flip = rng.integers(0, 1 << 24, len(paints)).astype(np.uint32)
    paints[solid, 1] ^= flip[solid]
    cap.buffers["paints"] = paints.tobytes()
    for t in cap.textures:
        a = np.frombuffer(t.rgba, np.uint8).reshape(-1, 4).astype(np.uint16)
        keep = rng.integers(128, 256, (1, 4)).astype(np.uint16)
        keep[0, 3] = 255
        t.rgba = (a * keep // 255).astype(np.uint8).tobytes()
    return cap


def _captures(case, seed):
    capture, _, S = _package()
    rng = np.random.default_rng(seed)
    n = case["frames"]
    if case["scene"] in RECORDED:
        names = RECORDED[case["scene"]]
        return [_recorded(capture, names[i % len(names)], rng, case.get("shift", 8))
                for i in range(n)]
    lib, caps = _planner(), []
    sizes = np.random.default_rng(n)  # the frames of a batch are of uneven size, the same for every seed
    for _ in range(n):
        w, h, p = case["width"], case["height"], case["paths"]
        if n > 1:
            w, h = (max(64, int(v * math.exp(sizes.uniform(-.5, .5)))) for v in (w, h))
            p = max(5, int(p * math.exp(sizes.uniform(-.7, .7))))
        if case["scene"] == "ui":
            sc = ui_scene(S, rng, w, h, p)
        elif case["scene"] == "plain":
            sc = S.plain_canvas(rng, w, h, p)
        elif case["scene"] == "full":
            sc = S.full_feature(seed=int(rng.integers(1 << 30)), width=w, height=h, n_paths=p)
        else:
            sc = S.stroke_stress(seed=int(rng.integers(1 << 30)), width=w, height=h, n_strokes=p)
        caps.append(_plan(lib, capture, sc.to_bytes()))
    return caps


# ---- the calls --------------------------------------------------------------


class State:
    """What a program has before the call: its context, its frames' records
    and targets, and its launch descriptions (or its graphs)."""


def _device_buffers(capture, rive_cuda, cap, keep):
    bufs = rive_cuda.DeviceBuffers()
    for name in capture.BUFFER_NAMES:
        b = cap.buffers.get(name, b"")
        if b:
            t = torch.from_numpy(np.frombuffer(b, np.uint8).copy()).cuda()
            keep.append(t)
            setattr(bufs, name, t.data_ptr())
    return bufs


def prepare(case, seed):
    capture, rive_cuda, _ = _package()
    s = State()
    s.call = case["call"]
    s.caps = _captures(case, seed)
    s.ctx = rive_cuda.Context(0)
    if case.get("queue"):
        s.ctx.set_raster_queue(True)
    if s.call == "app":
        s.target = s.ctx.render_target(s.caps[0].width, s.caps[0].height)
        return s
    s.keep = []
    s.bufs = [_device_buffers(capture, rive_cuda, c, s.keep) for c in s.caps]
    s.targets = [torch.zeros((c.height, c.width, 4), dtype=torch.uint8, device="cuda")
                 for c in s.caps]
    if s.call in ("device", "noalloc"):
        s.descs = []
        for c, b, t in zip(s.caps, s.bufs, s.targets):
            for f in c.flushes:
                d, k = s.ctx.desc_for(f) if s.call == "device" else rive_cuda.make_desc(f)
                s.keep.append(k)
                s.descs.append((f, d, b, t.data_ptr()))
        return s
    # Logical flush i of every frame that has one; a frame's later flushes load
    # what its earlier ones wrote.
    s.waves, s.graphs = [], []
    for i in range(max(len(c.flushes) for c in s.caps)):
        items = [(c.flushes[i], b, t.data_ptr())
                 for c, b, t in zip(s.caps, s.bufs, s.targets) if i < len(c.flushes)]
        if s.call == "graph":
            s.graphs.append(s.ctx.graph(items))
            continue
        arr = (rive_cuda.BatchFlush * len(items))()
        for k, (f, b, p) in enumerate(items):
            d, keep = s.ctx.desc_for(f)
            s.keep.append((d, keep))
            arr[k].desc = ctypes.cast(ctypes.pointer(d), ctypes.c_void_p)
            arr[k].buffers = b
            arr[k].target_pixels_device = p
        s.waves.append(arr)
    return s


def run(state):
    s = state
    ctx, lib = s.ctx, s.ctx.lib
    if s.call == "app":
        return ctx.render(s.caps[0], s.target)
    if s.call == "device":
        for _, d, b, t in s.descs:
            ctx.check(lib.rive_cuda_flush_device(ctx.h, ctypes.byref(d), ctypes.byref(b),
                                                 ctypes.c_void_p(t), None), "flush_device")
    elif s.call == "noalloc":
        err = ctypes.create_string_buffer(256)
        for _, d, b, t in s.descs:
            ctx.check(lib.rive_cuda_flush_device_noalloc(
                ctypes.byref(d), ctypes.byref(b), ctypes.c_void_p(t), None, err, 256),
                "flush_device_noalloc")
    elif s.call == "batch":
        for arr in s.waves:
            ctx.check(lib.rive_cuda_flush_batch(ctx.h, arr, len(arr), None), "flush_batch")
    else:
        # Several graphs of one frame list run in order on one stream.
        stream = torch.cuda.current_stream().cuda_stream if len(s.graphs) > 1 else None
        for g in s.graphs:
            g.launch(stream)
    return s.targets


# Per path: tessellated segments, the bytes of its records, and the pixels it
# covers as a share of its frame (or in pixels) -- averages of each scene kind.
SHAPES = {
    "ui": (370, 2400, None, 9000),
    "plain": (800, 800, 0.3, None),
    "full": (3100, 8350, None, 9500),
    "strokes": (290, 1380, None, 6500),
}
RECORDED_WORK = {  # pixels, record bytes, tessellated vertices of one frame
    "feathered": (1166400, 548000, 36900),
    "images": (862544, 120000, 12000),
    "mix": (1653000, 154000, 27300),
}


def work(case):
    """Records read once, target pixels written once; per tessellated vertex
    about 150 operations, per covered pixel and path about 40."""
    n = case["frames"]
    if case["scene"] in RECORDED:
        px, rec, verts = RECORDED_WORK[case["scene"]]
        return {"bytes": n * (px * 4 + rec), "flops": n * (verts * 150.0 + px * 3 * 40.0)}
    px, p = case["width"] * case["height"], case["paths"]
    segs, rec, share, area = SHAPES[case["scene"]]
    covered = p * (px * share if share else min(area, px))
    return {"bytes": n * (px * 4 + p * rec), "flops": n * (p * segs * 150.0 + covered * 40.0)}


def exact(case, seed):
    """The targets are RGBA8 bytes: they have no value beside their own."""
    return None
