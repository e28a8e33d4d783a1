"""Which pixels the raster gives a triangle, against the edge rule evaluated
pixel by pixel in numpy: every (triangle, pixel) decision must agree exactly.

The triangles are interior triangles (opaque, undithered, one path each), so a
pixel's colour names the last triangle that covers it. An edge's value is
E = fma(A, x, fma(B, y, C)) with C = fma(A, dx, B dy) at the tile's first pixel
centre; with coordinates on the 1/256-pixel grid all exact values here are
multiples of 2^-16 below 2^33, so float64 holds them exactly and one rounding
to float32 restates each fused step."""
import numpy as np
import pytest

from conftest import device_buffers, load_golden, load_package

load_package()
# Ragged at every tile size. "wide": more than kWideTiles tiles of 8 and of 16
# pixels, so its largest triangles are binned strip by strip.
SIZES = {"ties": (331, 203), "slivers": (331, 203), "small": (331, 203), "wide": (701, 475)}


def triangles(kind, n, rng):
    """n clockwise (y down) triangles, (n, 3, 2) on the 1/256-pixel grid."""
    W, H = SIZES[kind]
    if kind == "ties":  # corners on and half-way between pixel centres, axis-aligned edges
        p = (rng.integers(-4, 2 * max(W, H) + 4, (n, 1, 2)) + rng.integers(-50, 50, (n, 3, 2))) / 2.0
        p[::3, 1, 1] = p[::3, 0, 1]
        p[1::3, 2, 0] = p[1::3, 1, 0]
    elif kind == "slivers":  # long and thin, far outside the canvas, rounded edge values
        a = rng.integers(-2000 * 256, 2400 * 256, (n, 1, 2)) / 256.0
        b = rng.integers(-2000 * 256, 2400 * 256, (n, 1, 2)) / 256.0
        p = np.concatenate([a, b, b + rng.integers(-300, 300, (n, 1, 2)) / 256.0], 1)
    elif kind == "wide":  # most of the canvas, and slivers across it
        p = rng.integers(-200 * 256, 900 * 256, (n, 3, 2)) / 256.0
        p[::4, 2] = p[::4, 1] + rng.integers(-900, 900, (len(p[::4]), 2)) / 256.0
    else:  # "small": a few pixels
        p = rng.integers(0, max(W, H) * 256, (n, 1, 2)) + rng.integers(-1400, 1400, (n, 3, 2))
        p = p / 256.0
    u, v = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    area = u[:, 0] * v[:, 1] - v[:, 0] * u[:, 1]
    p[area < 0] = p[area < 0][:, [0, 2, 1]]
    return p


def f32(x):
    return np.asarray(x, np.float64).astype(np.float32).astype(np.float64)


def expected(tris, tile, W, H):
    """Per pixel the last covering triangle's number + 1, or 0."""
    out = np.zeros((H, W), np.int64)
    for i, p in enumerate(tris):
        u, v = p[1] - p[0], p[2] - p[0]
        if u[0] * v[1] - v[0] * u[1] <= 0:
            continue
        lo = np.maximum(np.ceil(p.min(0) - .5), 0)
        hi = np.minimum(np.floor(p.max(0) - .5) + 1, (W, H))
        if (lo >= hi).any():
            continue
        ly0, lx0 = (lo[::-1] // 8 * 8).astype(int)  # whole 8x4 blocks about the pixel box
        ly1, lx1 = (-(-hi[::-1] // 8) * 8).astype(int)
        ys, xs = np.mgrid[ly0:min(ly1, H), lx0:min(lx1, W)]
        ox, oy = xs // tile * tile, ys // tile * tile
        lx, ly = xs - ox, ys - oy
        bx, by = lx // 8 * 8, ly // 4 * 4  # the pixel's 8x4 block in its tile
        # The part of the block inside the pixel box, tile-local, empty or not.
        x0, x1 = np.maximum(lo[0] - ox, bx), np.minimum(hi[0] - ox, bx + 8)
        y0, y1 = np.maximum(lo[1] - oy, by), np.minimum(hi[1] - oy, by + 4)
        inside = (x0 < x1) & (y0 < y1)
        for k in range(3):
            a, b = p[k], p[(k + 1) % 3]
            first, last = (a, b) if (a[1], a[0]) < (b[1], b[0]) else (b, a)
            A, B = -(b[1] - a[1]), b[0] - a[0]
            assert first is not last
            C = f32(A * (ox + .5 - first[0]) + f32(B * (oy + .5 - first[1])))
            E = A * lx + f32(B * ly + C)
            edge_in = A > 0 or (A == 0 and B > 0)
            # The block's corner that maximises E must not be outside.
            corner = A * (x1 - 1 if A > 0 else x0) + f32(B * (y1 - 1 if B > 0 else y0) + C)
            inside &= ((E >= 0) if edge_in else (E > 0)) & (corner >= 0)
        out[ys[inside], xs[inside]] = i + 1
    return out


def flush_of(tris, path_ids, W, H):
    """A capture of one batch of interior triangles, and its device buffers."""
    n, paths_n = len(tris), int(path_ids.max())
    cap = load_golden("tri_fills_s21")[0]  # for a FlushUniforms record and a descriptor
    f = cap.flushes[0]
    paths = np.zeros((paths_n + 1, 16), np.float32)
    paths[1:, 0] = paths[1:, 3] = 1.0
    paints = np.zeros((paths_n + 1, 2), np.uint32)
    paints[:, 0] = 1  # solid
    paints[:, 1] = np.arange(paths_n + 1, dtype=np.uint32) | 0xFF000000
    verts = np.zeros((n, 3, 3), np.uint32)
    verts[..., :2] = tris.astype(np.float32).view(np.uint32)
    verts[..., 2] = path_ids[:, None].astype(np.uint32) | 0x10000  # weight 1
    cap.buffers = {"flush_uniforms": cap.buffers["flush_uniforms"], "paths": paths.tobytes(),
                   "paints": paints.tobytes(), "paint_aux": bytes(128 * (paths_n + 1)),
                   "triangles": verts.tobytes()}
    f.desc.update(render_target_width=W, render_target_height=H, ub2=W, ub3=H,
                  path_count=paths_n + 1, contour_count=0, tess_span_count=0, tess_data_height=0,
                  dither_mode=0, color_clear_value=0xFF000000, combined_shader_features=0)
    f.batches = np.array([[3, 3 * n, 0, 0, 16, 0, 3, 0]], np.uint32)
    return f, device_buffers(cap)


def render(f, bufs, W, H, tile=16, queue=False):
    """The image as (H, W) path numbers, and the flush's statistics."""
    import torch
    from rive_runtime_gb300 import rive_cuda
    ctx = rive_cuda.Context(0)
    ctx.set_raster_config(tile)
    ctx.set_raster_queue(queue)
    target = torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda")
    ctx.flush_device(f, bufs, target.data_ptr())
    ctx.sync()
    img = target.cpu().numpy().astype(np.int64)
    stats = ctx.stats()
    ctx.close()
    return img[..., 0] | (img[..., 1] << 8) | (img[..., 2] << 16), stats


@pytest.mark.gpu
@pytest.mark.parametrize("queue", [False, True])
@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("kind,n", [("ties", 700), ("slivers", 700), ("small", 3000), ("wide", 80)])
def test_covered_pixels_are_exact(kind, n, tile, queue):
    if queue and tile != 16:
        pytest.skip("the work queue takes 16-pixel tiles")
    W, H = SIZES[kind]
    tris = triangles(kind, n, np.random.default_rng(7))
    f, (bufs, keep) = flush_of(tris, np.arange(1, n + 1), W, H)
    got, _ = render(f, bufs, W, H, tile, queue)
    want = expected(tris, tile, W, H)
    assert (want > 0).mean() > .02
    assert np.array_equal(got, want), np.argwhere(got != want)[:5]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 16383, 16384, 16400])
def test_wide_triangles_around_the_capacity_of_their_list(n):
    """Canvas-wide triangles, as many as the binner sets aside (kWideCapacity)
    and some more, which it walks in place: every one has every tile."""
    W, H = 16 * 33, 16 * 32
    tris = np.tile(np.array([[[-10, -10], [3000, -10], [-10, 3000]]], np.float64), (n, 1, 1))
    f, (bufs, keep) = flush_of(tris, np.full(n, 1), W, H)
    got, stats = render(f, bufs, W, H)
    assert stats["bin_entries"] == n * 33 * 32
    assert (got == 1).all()


@pytest.mark.gpu
@pytest.mark.parametrize("W,H", [(128, 120), (640, 470)])  # one and two key bytes
@pytest.mark.parametrize("n", [1, 1023, 8192, 8193, 131072, 131073, 262144, 262145])
def test_bins_at_the_edges_of_the_one_cluster_passes(n, W, H):
    """n triangles of one bin entry each, around the sizes at which the scan and
    the sort of small frames change their share per thread or give way to the
    library's: alone, and in a batch too large for either, the same image."""
    import torch
    from rive_runtime_gb300 import rive_cuda
    rng = np.random.default_rng(n)
    at = np.stack([rng.integers(0, W // 16, n), rng.integers(0, H // 16, n)], 1) * 16.0
    at += rng.integers(0, 10, (n, 2))
    tris = at[:, None] + np.array([[0, 0], [5.5, 0], [0, 5.5]])
    ids = 1 + np.arange(n) * min(n, 60000) // n
    f, (bufs, keep) = flush_of(tris, ids, W, H)
    got, stats = render(f, bufs, W, H)
    assert stats["bin_entries"] == n and stats["triangles"] == n
    m = 300000
    filler, (fbufs, fkeep) = flush_of(np.tile(tris[:1], (m, 1, 1)), np.full(m, 1), W, H)
    targets = [torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda") for _ in range(2)]
    ctx = rive_cuda.Context(0)
    ctx.flush_batch([(f, bufs, targets[0].data_ptr()), (filler, fbufs, targets[1].data_ptr())])
    ctx.sync()
    img = targets[0].cpu().numpy().astype(np.int64)
    ctx.close()
    assert np.array_equal(got, img[..., 0] | (img[..., 1] << 8) | (img[..., 2] << 16))
    # The pixel (1, 1) of the last triangle has its colour.
    x, y = at[-1].astype(int) + 1
    assert got[y, x] == ids[-1]


@pytest.mark.gpu
@pytest.mark.parametrize("W,H", [(640, 470), (4112, 4112)])  # 16 and 32-bit keys
@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 9, 255, 1025, 140000])
def test_tile_ranges_at_the_edges_of_a_load(n, W, H):
    """n one-entry triangles in a batch whose keys take the vectorised range
    pass (a filler scene brings the entries past the one-cluster sort, or the
    canvas the tiles past 16-bit keys)."""
    import torch
    from rive_runtime_gb300 import rive_cuda
    rng = np.random.default_rng(n)
    at = np.stack([rng.integers(0, W // 16, n), rng.integers(0, H // 16, n)], 1) * 16.0
    at[-1] = [W // 16 * 16 - 16, H // 16 * 16 - 16]  # the last full tile
    tris = at[:, None] + np.array([[1, 1], [6.5, 1], [1, 6.5]])
    ids = 1 + np.arange(n) * min(n, 60000) // n
    f, (bufs, keep) = flush_of(tris, ids, W, H)
    m = 1 if W > 1000 else 140000
    filler, (fbufs, fkeep) = flush_of(np.tile(tris[:1], (m, 1, 1)), np.full(m, 1), W, H)
    targets = [torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda") for _ in range(2)]
    ctx = rive_cuda.Context(0)
    ctx.flush_batch([(filler, fbufs, targets[0].data_ptr()), (f, bufs, targets[1].data_ptr())])
    ctx.sync()
    img = targets[1].cpu().numpy().astype(np.int64)
    ctx.close()
    got = img[..., 0] | (img[..., 1] << 8) | (img[..., 2] << 16)
    # Every tile's shape has the colour of the last triangle there.
    want = {tuple(p): i for p, i in zip(at.astype(int), ids)}
    assert all(got[y + 2, x + 2] == i for (x, y), i in want.items())
    assert (got > 0).sum() == len(want) * (got[H // 16 * 16 - 16:, W // 16 * 16 - 16:] > 0).sum()


def test_unorm_float_is_the_correctly_rounded_quotient():
    """kUnormHi / kUnormLo of kernels_raster.cu: b / 255 for every byte by one
    rounded product and one fused step (float64 holds both exactly)."""
    hi, lo = np.float64(float.fromhex("0x1.010102p-8")), np.float64(float.fromhex("-0x1.fdfdfep-33"))
    b = np.arange(256, dtype=np.float64)
    got = (b * hi + f32(b * lo)).astype(np.float32)
    assert np.array_equal(got, np.arange(256, dtype=np.float32) / np.float32(255))


@pytest.mark.gpu
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("name", ["plain_small_s1", "stroke_stress_s5", "strokes_s3"])
def test_patches_three_a_warp_match_one_a_warp(name, mixed):
    """A flush small enough for a warp per patch, and as many copies of it as
    make a batch whose warps shade three patches at once: the same images.
    "mixed": every third span takes another contour's number, so patches hold
    vertices of several contours, of fills beside strokes."""
    import torch
    from rive_runtime_gb300 import rive_cuda
    cap = load_golden(name)[0]
    f = cap.flushes[0]
    b = f.batches = np.array(f.batches)
    b[:, 1] = np.minimum(b[:, 1], 8191)  # of plain_small_s1, the first half of its patches
    if mixed:
        spans = np.frombuffer(cap.buffers["tess_spans"], np.uint32).reshape(-1, 16).copy()
        rng = np.random.default_rng(5)
        other = rng.integers(1, f.desc["contour_count"] + 1, len(spans[::3])).astype(np.uint32)
        spans[::3, 15] = (spans[::3, 15] & 0xffff0000) | other
        cap.buffers["tess_spans"] = spans.tobytes()
    bufs, keep = device_buffers(cap)
    copies = 8192 // int(b[:, 1].sum()) + 2
    targets = [torch.zeros((cap.height, cap.width, 4), dtype=torch.uint8, device="cuda")
               for _ in range(copies + 1)]
    ctx = rive_cuda.Context(0)
    ctx.flush_device(f, bufs, targets[0].data_ptr())
    ctx.sync()
    ctx.flush_batch([(f, bufs, t.data_ptr()) for t in targets[1:]])
    ctx.sync()
    ctx.close()
    want = targets[0].cpu().numpy()
    assert len(np.unique(want.reshape(-1, 4), axis=0)) > 20
    for t in targets[1:]:
        assert np.array_equal(t.cpu().numpy(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("queue", [False, True])
@pytest.mark.parametrize("tiles", [8191, 8192, 8193, 65600])  # one and two launches, 16 and 32-bit keys
def test_tiles_split_between_raster_variants(tiles, queue):
    """Feathered, atlas, image and plain frames, and a plain canvas that brings
    the batch to `tiles` tiles: the images of single flushes."""
    import torch
    from conftest import render_one_by_one
    from rive_runtime_gb300 import rive_cuda
    names = ["feathered_s33", "feather_atlas_s35", "images_s41", "clips_s13", "feather_strokes_s31"]
    caps = [load_golden(n)[0] for n in names]
    pairs = [device_buffers(c) for c in caps]
    bufs = [p[0] for p in pairs]
    rest = tiles - sum(((c.width + 15) // 16) * ((c.height + 15) // 16) for c in caps)
    W, H = 16 * (rest if rest < 4000 else rest // 64), 16 * (1 if rest < 4000 else 64)
    odd = rest - (W // 16) * (H // 16)  # and what is left of it
    sizes = [(W, H)] + ([(16 * odd, 16)] if odd else [])
    rng = np.random.default_rng(9)
    plain = []
    for w, h in sizes:
        at = np.stack([rng.integers(0, w // 16, 3000), rng.integers(0, h // 16, 3000)], 1) * 16.0
        tris = at[:, None] + np.array([[1, 1], [14.5, 2], [3, 12.5]])
        f, (b, keep) = flush_of(tris, np.arange(1, 3001), w, h)
        plain.append((f, b, keep, w, h, render(f, b, w, h)[0]))
    ctx = rive_cuda.Context(0)
    stream = torch.cuda.current_stream().cuda_stream
    want = render_one_by_one(ctx, caps, bufs, stream)
    ctx.set_raster_queue(queue)
    targets = [torch.zeros((c.height, c.width, 4), dtype=torch.uint8, device="cuda") for c in caps]
    ptargets = [torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda") for _, _, _, w, h, _ in plain]
    assert all(len(c.flushes) == 1 for c in caps)
    items = [(c.flushes[0], b, t.data_ptr()) for c, b, t in zip(caps, bufs, targets)]
    items[2:2] = [(f, b, t.data_ptr()) for (f, b, _, _, _, _), t in zip(plain, ptargets)]
    for call in ("batch", "graph"):
        for t in targets + ptargets:
            t.fill_(7)
        if call == "batch":
            ctx.flush_batch(items, stream)
            ctx.sync(stream)
        else:
            g = ctx.graph(items)
            for _ in range(2):
                g.launch(stream)
            g.check(stream)
            g.close()
        torch.cuda.synchronize()
        for n, t, w in zip(names, targets, want):
            assert np.array_equal(t.cpu().numpy(), w), (call, n)
        for (_, _, _, _, _, w), t in zip(plain, ptargets):
            img = t.cpu().numpy().astype(np.int64)
            assert np.array_equal(img[..., 0] | (img[..., 1] << 8) | (img[..., 2] << 16), w), call
    ctx.close()


@pytest.mark.gpu
# Flushes of 16,384 spans on are tessellated by warps of 8 spans, of 65,536 on by
# warps of 16 where a span has few texels.
@pytest.mark.parametrize("name,spans", [
    ("stroke_stress_s5", 16384), ("stroke_stress_s5", 66000), ("plain_small_s1", 16500),
    ("full_odd_s11", 17000), ("feather_strokes_s31", 16390), ("silver_police_files_f60", 66000),
    ("silver_rewards_f10", 66000)])
def test_spans_by_warps_match_spans_by_lanes(name, spans):
    """A flush's spans, and as many copies of them (each in rows of its own) as
    take the packed tessellation: every copy has the same texels."""
    import torch
    from conftest import tess_written
    from rive_runtime_gb300 import rive_cuda
    cap = load_golden(name)[0]
    f = cap.flushes[0]
    d = f.desc
    h, first, n = d["tess_data_height"], d["first_tess_span"], d["tess_span_count"]
    written = tess_written(cap, 0)
    ctx = rive_cuda.Context(0)
    target = torch.zeros((cap.height, cap.width, 4), dtype=torch.uint8, device="cuda")

    def texels(height):
        bufs, keep = device_buffers(cap)
        ctx.flush_device(f, bufs, target.data_ptr())
        ctx.sync()
        t = np.asarray(ctx.read_tess(height)).view(np.uint32).reshape(-1, 4)
        return t.reshape(-1, 2048 * h, 4)[:, written], target.cpu().numpy()

    want, image = texels(h)
    one = np.frombuffer(cap.buffers["tess_spans"], np.uint32).reshape(-1, 16)[first:first + n]
    copies = -(-spans // n)
    all_spans = np.tile(one, (copies, 1, 1)).reshape(copies, n, 16)
    for i in range(copies):
        y = all_spans[i, :, 10:12].copy().view(np.float32) + np.float32(i * h)
        all_spans[i, :, 10:12] = y.view(np.uint32)
    cap.buffers["tess_spans"] = all_spans.tobytes()
    d.update(first_tess_span=0, tess_span_count=copies * n, tess_data_height=copies * h)
    got, image2 = texels(copies * h)
    ctx.close()
    assert len(got) == copies
    for g in got:
        assert np.array_equal(g, want[0])
    assert np.array_equal(image, image2)
