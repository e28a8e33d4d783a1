"""Records and settings at the edge of what the kernels take: each against the
oracle, or against exactly sized, unlimited renders that are themselves held to
it by the golden tests."""
import numpy as np
import pytest

from conftest import device_buffers, load_golden, load_package

load_package()


@pytest.mark.gpu
@pytest.mark.parametrize("copies", [1, 20])  # spans by lanes, and packed in warps
@pytest.mark.parametrize("name", ["strokes_s3", "full_odd_s11"])
def test_spans_without_vertices_have_the_shaders_texels(name, copies):
    """Spans whose three counts are zero: their vertex total wraps to 2^32 - 1,
    and their texels are what the shader's arithmetic gives for it."""
    import oracle
    from conftest import tess_written
    from rive_runtime_gb300 import rive_cuda
    cap = load_golden(name)[0]
    f = cap.flushes[0]
    d = f.desc
    h, first, n = d["tess_data_height"], d["first_tess_span"], d["tess_span_count"]
    spans = np.frombuffer(cap.buffers["tess_spans"], np.uint32).reshape(-1, 16)
    one = spans[first:first + n].copy()
    one[np.random.default_rng(3).random(n) < .2, 14] = 0
    # Beyond 128 texels float32 spaces the index by 256: a span across two whole
    # rows of its own, and one that starts left of them.
    long = np.repeat(one[:1], 2, axis=0)
    long[:, 14] = 0
    long[:, 10:12] = np.array([[h, h + 1], [h + 2, h + 3]], np.float32).view(np.uint32)
    long[:, 12:14] = [[2048 << 16, 2048], [2000 << 16 | (-30 & 0xffff), -30 << 16 & 0xffffffff | 2000]]
    one, n, h = np.concatenate([one, long]), n + 2, h + 4
    cap.buffers["tess_spans"] = one.tobytes()
    d.update(first_tess_span=0, tess_span_count=n, tess_data_height=h)
    written = tess_written(cap, 0)
    want = oracle.tessellate(cap)[written]
    assert (one[:, 14] == 0).sum() > 8
    many = np.tile(one, (copies, 1, 1))
    for i in range(copies):
        many[i, :, 10:12] = (one[:, 10:12].view(np.float32) + np.float32(i * h)).view(np.uint32)
    cap.buffers["tess_spans"] = many.tobytes()
    d.update(tess_span_count=copies * n, tess_data_height=copies * h)
    assert copies == 1 or copies * n >= 16384
    ctx = rive_cuda.Context(0)
    import torch
    target = torch.zeros((cap.height, cap.width, 4), dtype=torch.uint8, device="cuda")
    bufs, keep = device_buffers(cap)
    ctx.flush_device(f, bufs, target.data_ptr())
    ctx.sync()
    got = np.asarray(ctx.read_tess(copies * h)).view(np.uint32).reshape(copies, 2048 * h, 4)
    ctx.close()
    for g in got:
        g = g[written]
        assert np.array_equal(g[:, 3], want[:, 3])
        a, b = g[:, :3].copy().view(np.float32), want[:, :3].copy().view(np.float32)
        assert ((a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))).all()


def parity(got, want):
    d = np.abs(got.astype(np.int16) - want.astype(np.int16)).max(axis=2)
    assert (d <= 2).mean() >= .999 and d.max() <= 8, (float((d <= 2).mean()), int(d.max()))


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.nan, -np.inf, -3e38])
@pytest.mark.parametrize("name,where", [(n, w) for n in ("strokes_s3", "feather_atlas_s35", "images_s41")
                                        for w in ("v", "span", "image") if w != "image" or n == "images_s41"])
def test_paints_that_are_not_finite(name, where, value):
    """Gradients whose row or span is not finite, image matrices likewise: a
    pixel of no coverage is written, too, and its colour is not the
    destination's (0 times NaN)."""
    import oracle
    from rive_runtime_gb300 import rive_cuda
    cap = load_golden(name)[0]
    paints = np.frombuffer(cap.buffers["paints"], np.uint32).reshape(-1, 2).copy()
    aux = np.frombuffer(cap.buffers["paint_aux"], np.float32).reshape(-1, 32).copy()
    n = min(len(paints), len(aux))
    gradient = np.isin(paints[:n, 0] & 15, (2, 3))
    image = (paints[:n, 0] & 0x800) != 0
    hit = np.flatnonzero(image if where == "image" else gradient)[::2]
    assert len(hit)
    if where == "v":
        paints[hit, 1] = np.float32(value).view(np.uint32)
    elif where == "span":
        aux[hit, 6:8] = 0, value
    else:
        aux[hit, 20] = value
    cap.buffers["paints"], cap.buffers["paint_aux"] = paints.tobytes(), aux.tobytes()
    ctx = rive_cuda.Context(0)
    got = ctx.render(cap)
    ctx.close()
    parity(got, oracle.render(cap))


@pytest.mark.gpu
def test_split_raster_under_the_limits_of_two_contexts():
    """A frame whose tiles are split between two launches, by contexts with
    different limits of resident CTAs in turn, single and as graphs: each keeps
    its own."""
    import oracle
    import torch
    from rive_runtime_gb300 import rive_cuda
    cap = load_golden("silver_bankcard_f10")[0]
    want = oracle.render(cap)
    bufs, keep = device_buffers(cap)
    stream = torch.cuda.Stream().cuda_stream
    made = []
    for ctas in (1, 4, 2, 0):
        ctx = rive_cuda.Context(0)
        ctx.set_raster_config(16, ctas)
        target = torch.zeros((cap.height, cap.width, 4), dtype=torch.uint8, device="cuda")
        made.append((ctx, target, ctx.graph([(cap.flushes[0], bufs, target.data_ptr())])))
    for ctx, target, graph in made + made:
        parity(ctx.render(cap), want)
        target.zero_()
        torch.cuda.synchronize()
        graph.launch(stream)
        graph.check(stream)
        parity(target.cpu().numpy(), want)
    for ctx, _, graph in made:
        graph.close()
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["strokes_s3", "clips_s13"])
def test_noalloc_in_a_second_cuda_context(name):
    """The no-allocation flush in a CUDA context made after the library has run
    in the device's primary one, where the one-cluster passes' function
    attributes were set: they hold in the other context as well."""
    import ctypes
    import oracle
    import torch
    from rive_runtime_gb300 import rive_cuda
    from rive_runtime_gb300.capture import BUFFER_NAMES
    cap = load_golden(name)[0]
    bufs, keep = device_buffers(cap)
    first = torch.zeros((cap.height, cap.width, 4), dtype=torch.uint8, device="cuda")
    rive_cuda.flush_device_noalloc(cap.flushes[0], bufs, first.data_ptr(), 0)
    torch.cuda.synchronize()
    cu = ctypes.CDLL("libcuda.so.1")

    def call(f, *args):
        assert getattr(cu, f)(*args) == 0, f

    call("cuCtxCreate_v2", ctypes.byref(ctypes.c_void_p()), 0, 0)
    try:
        def alloc(data):
            p = ctypes.c_uint64()
            call("cuMemAlloc_v2", ctypes.byref(p), ctypes.c_size_t(max(len(data), 16)))
            call("cuMemcpyHtoD_v2", p, data, ctypes.c_size_t(len(data)))
            return p.value

        bufs2 = rive_cuda.DeviceBuffers()
        for n in BUFFER_NAMES:
            data = cap.buffers.get(n, b"")
            setattr(bufs2, n, alloc(data) if data else None)
        target = alloc(bytes(4 * cap.width * cap.height))
        rive_cuda.flush_device_noalloc(cap.flushes[0], bufs2, target, 0)
        got = np.zeros((cap.height, cap.width, 4), np.uint8)
        call("cuMemcpyDtoH_v2", got.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint64(target),
             ctypes.c_size_t(got.nbytes))
    finally:
        old = ctypes.c_void_p()
        call("cuCtxPopCurrent_v2", ctypes.byref(old))
        call("cuCtxDestroy_v2", old)
    assert np.array_equal(got, first.cpu().numpy())
    parity(got, oracle.render(cap))


@pytest.mark.gpu
def test_kernel_launches_are_counted():
    """flush_stats.kernel_launches: the library's own kernels of the last flush,
    where a setting or a size adds one."""
    import torch
    from rive_runtime_gb300 import rive_cuda
    ctx = rive_cuda.Context(0)
    ctx.set_bin_speculation(False)

    def launches(cap):
        ctx.render(cap)
        return ctx.stats()["kernel_launches"]

    small = load_golden("strokes_s3")[0]  # with gradients, 256 tiles
    # Preparation, tessellation with ramps, set-up, scan, binner, sort, raster.
    assert launches(small) == 7
    bufs, keep = device_buffers(small)
    target = torch.zeros((small.height, small.width, 4), dtype=torch.uint8, device="cuda")
    graph = ctx.graph([(small.flushes[0], bufs, target.data_ptr())])
    assert graph.stats()["kernel_launches"] == 7
    graph.close()
    ctx.set_raster_queue(True)
    assert launches(small) == 8  # and the tiles' order
    ctx.set_raster_queue(False)
    ctx.set_profiling(True)
    assert launches(small) == 8  # and the ramps by themselves
    ctx.set_profiling(False)
    ctx.set_bin_speculation(True)
    assert launches(small) == 7
    ctx.set_bin_speculation(False)
    # 15,645 tiles: set-up passes of fans, center-AA fans, triangles; the wide
    # triangles' count; the atlas; two rasters.
    large = load_golden("silver_bankcard_f10")[0]
    split = launches(large)
    ctx.set_raster_config(32)
    assert launches(large) == split - 1
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("queue", [False, True])
@pytest.mark.parametrize("name", ["silver_bankcard_f10", "silver_rewards_atlas_f10",
                                  "silver_police_files_f60", "full_odd_s11"])
def test_overflowing_speculation_against_the_oracle(name, queue):
    """Frames whose tiles are split, ordered or chained, flushed on bins that a
    far smaller frame sized: the back half runs again over the same tile heads."""
    import oracle
    from rive_runtime_gb300 import rive_cuda
    cap = load_golden(name)[0]
    ctx = rive_cuda.Context(0)
    ctx.set_raster_queue(queue)
    ctx.render(load_golden("mesh_overlap")[0])
    got = ctx.render(cap)
    first = ctx.stats()
    again = ctx.render(cap)
    assert ctx.stats()["kernel_launches"] < first["kernel_launches"]  # the first ran twice
    assert ctx.stats()["bin_entries"] == first["bin_entries"]
    ctx.close()
    parity(got, oracle.render(cap))
    assert np.array_equal(got, again)


@pytest.mark.gpu
def test_contexts_on_threads_against_the_oracle():
    """Small chained frames and a split one, each by a thread with a context of
    its own, at the same time."""
    import threading
    import oracle
    from rive_runtime_gb300 import rive_cuda
    names = ["strokes_s3", "feathered_s33", "clips_s13", "silver_bankcard_f10"]
    caps = [load_golden(n)[0] for n in names]
    images = [[] for _ in caps]

    def work(i):
        ctx = rive_cuda.Context(0)
        for _ in range(15):
            images[i].append(ctx.render(caps[i]))
        ctx.close()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(caps))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for cap, got in zip(caps, images):
        assert len(got) == 15
        parity(got[0], oracle.render(cap))
        assert all(np.array_equal(g, got[0]) for g in got)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["clips_s13", "image_meshes_s43"])
def test_new_memory_is_clear_before_it_is_used(name):
    """Targets and render buffers made and used while the legacy default stream is
    busy: their clears neither wait for it nor come after the flush."""
    import torch
    from rive_runtime_gb300 import rive_cuda
    cap, warm = load_golden(name)[0], load_golden(name)[0]
    ctx = rive_cuda.Context(0)
    want = ctx.render(warm)
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)  # on the legacy stream, about 0.1 s
    target = ctx.render_target(cap.width, cap.height)
    images = []
    for _ in range(2):
        ctx.upload_frame(cap)
        for f in cap.flushes:
            ctx.flush(f, target)
        ctx.sync()
        images.append(ctx.read_target(target, cap.width, cap.height))
        torch.cuda.synchronize()
        images.append(ctx.read_target(target, cap.width, cap.height))
    ctx.close()
    for image in images:
        assert np.array_equal(image, want)
