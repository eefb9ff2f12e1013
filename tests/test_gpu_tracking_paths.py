"""The tracking, pre-pass and display kernels at the sizes and scenes where
their special paths can go wrong, bit for bit against the oracle or the general
path: the march's jump through empty space, the persistent stages' common
parts, lights left out by a bound, transfer functions read by bucket, the
gradient maximum from cell means, quads and brick minima at ragged sizes, the
bilateral tiles, and batch windows of one view."""
import ctypes
import importlib

import numpy as np
import pytest

import oracle_lib as OL
from test_oracle_ref import random_scene

pytestmark = pytest.mark.gpu

C = OL.C
S = OL.PKG.scenes


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.fixture(scope="module")
def env():
    import torch
    assert torch.cuda.is_available(), "GPU tests need CUDA"
    lib = C.load_library()
    C.check(lib.er_set_device(0))
    yield torch, lib, importlib.import_module("exposure-render_gb300.runtime")
    lib.er_reset()


def gpu_sum(torch, r, spp, first=0):
    d = torch.zeros((r.height, r.width, 4), dtype=torch.float32, device="cuda")
    r.trace_sum_device(d.data_ptr(), spp, 0, first, 0, None)
    torch.cuda.synchronize()
    return d.cpu().numpy()


def check_sum(env, oracle, sc, spp=2):
    torch, lib, runtime = env
    r = runtime.Renderer(sc, lib)
    h = OL.SceneHandle(oracle, sc)
    try:
        assert np.array_equal(bits(gpu_sum(torch, r, spp)), bits(h.render_sum(spp, nthreads=8)))
    finally:
        r.close()
        h.close()


@pytest.mark.parametrize("engine", [0, 1], ids=["wavefront", "one-kernel"])
@pytest.mark.parametrize("seed", range(6))
def test_random_scenes_march(env, oracle, seed, engine):
    """random volumes, unsorted transfer-function nodes, lights of every shape"""
    sc = random_scene(seed)
    sc.tracer.settings.engine = engine
    check_sum(env, oracle, sc)


@pytest.mark.parametrize("brick,stages", [(1, 0), (2, 1), (3, 2), (8, 1), (8, 0), (64, 3)])
@pytest.mark.parametrize("seed", [1, 4])
def test_random_scenes_delta(env, oracle, seed, brick, stages):
    sc = random_scene(seed)
    s = sc.tracer.settings
    s.free_flight, s.mis, s.stratify, s.majorant_brick, s.tune_stages = 1, 1, 1, brick, stages
    check_sum(env, oracle, sc, spp=4)


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 2, 5), (4, 4, 4), (5, 4, 9), (17, 1, 33), (65, 8, 6)])
def test_march_map_ragged_volumes(env, oracle, shape):
    """volumes of a fraction of a map brick, a brick exactly, and one voxel more"""
    rng = np.random.default_rng(sum(shape))
    sc = S.scene_tiny(film=(24, 20), seed=3)
    v = rng.integers(0, 3000, size=shape).astype(np.uint16)
    v[rng.random(shape) < 0.6] = 0
    sc.volume = v
    check_sum(env, oracle, sc)


@pytest.mark.parametrize("nodes", [[(0.0, 0.0), (5000.0, 0.0)], [(0.0, 0.0), (300.0, -0.2), (900.0, 0.0), (2000.0, 0.5), (5000.0, 0.5)],
                                   [(0.0, 0.4), (60.0, 0.0), (5000.0, 0.0)]], ids=["empty", "negative", "air"])
def test_march_map_transfer_functions(env, oracle, nodes):
    """nothing opaque, a negative opacity (its sum falls: not empty), opaque air around empty matter"""
    sc = S.scene_tiny(res=24, film=(24, 20), seed=3)
    sc.tracer.opacity = C.make_plf(nodes)
    check_sum(env, oracle, sc)


@pytest.mark.parametrize("clip_far,aperture", [(1e9, 0.0), (1e12, 0.0), (1.9, 0.03)])
def test_lights_with_extreme_rays(env, oracle, clip_far, aperture):
    """rays whose end point the exact light tests cannot represent, and rays that end inside the volume"""
    sc = S.scene_objects(res=20, film=(24, 20))
    sc.tracer.camera.clip_far = clip_far
    sc.tracer.camera.aperture_size = aperture
    sc.tracer.camera.focal_distance = 2.0
    check_sum(env, oracle, sc)


def light_of(shape, pos, **kw):
    L = C.er_light_desc()
    L.visible = 1
    L.shape = S.make_shape(shape, S.look_at_tm(pos, (0.0, 0.0, 0.0), (0.0, 1.0, 0.0)), **kw)
    L.texture_id = 0
    L.multiplier = 4.0
    return L


LIGHTS = {"plane": (C.SHAPE_PLANE, (0.3, 1.1, 0.9), dict(size=(0.6, 0.4, 0.0))), "disk": (C.SHAPE_DISK, (-0.9, 0.5, 0.8), dict(outer=0.3)),
          "ring": (C.SHAPE_RING, (0.2, -0.9, 1.0), dict(inner=0.1, outer=0.3)), "sphere": (C.SHAPE_SPHERE, (0.8, 0.8, -0.6), dict(outer=0.2)),
          "around": (C.SHAPE_SPHERE, (0.0, 0.0, 1.0), dict(outer=5.0))}


@pytest.mark.parametrize("kind", list(LIGHTS))
@pytest.mark.parametrize("shadow,far,mult", [(0.0, None, 1), (1e-9, None, 1), (1e-7, None, 1), (1e-5, None, 1), (-1e-8, None, 1), (None, 0.0, 1),
                                             (None, 1e-9, 1), (0.0, None, 100)])
def test_lights_with_rays_of_no_length(env, oracle, kind, shadow, far, mult):
    """rays so short that their end rounds to their origin: the exact light and
    object tests divide zero by zero there and count flat shapes as hit"""
    shape, pos, kw = LIGHTS[kind]
    sc = S.scene_objects(res=20, film=(24, 20))
    sc.lights = [light_of(shape, tuple(mult * v for v in pos), **kw)]
    t = sc.tracer
    t.light_count, t.light_ids[0] = 1, 0
    if shadow is not None:
        t.settings.max_shadow_distance = shadow
    if far is not None:
        t.camera.clip_near, t.camera.clip_far = 0.0, far
    for delta in (0, 1):
        t.settings.free_flight = t.settings.mis = delta
        check_sum(env, oracle, sc)


@pytest.mark.parametrize("shape,spacing", [((1, 1, 1), (1, 1, 1)), ((2, 3, 1), (1, 1, 1)), ((31, 15, 29), (1, 1, 1)), ((33, 14, 30), (1, 1, 1)),
                                           ((64, 30, 61), (0.7, 0.7, 0.7)), ((20, 21, 22), (1.0, 2.0, 0.5))])
@pytest.mark.parametrize("kind", ["noise", "flat", "spike"])
def test_gradient_maximum_equals_the_full_pass(env, shape, spacing, kind):
    torch, lib, runtime = env
    rng = np.random.default_rng(7)
    v = {"noise": rng.integers(0, 65536, size=shape), "flat": np.full(shape, 1000), "spike": np.zeros(shape)}[kind].astype(np.uint16)
    if kind == "spike":
        v[tuple(n // 2 for n in shape)] = 40000
    sc = S.scene_tiny(film=(8, 8))
    sc.volume, sc.spacing = v, spacing
    r = runtime.Renderer(sc, lib)
    try:
        gm = torch.zeros(shape, dtype=torch.int16, device="cuda")
        full = r.gradient_magnitude(gm.data_ptr())
        assert r.gradient_magnitude() == full
    finally:
        r.close()


@pytest.mark.parametrize("shape", [(1, 1, 1), (33, 14, 30), (70, 61, 100)])
@pytest.mark.parametrize("kind", ["labels", "more labels", "smooth", "slope", "corner"])
def test_gradient_maximum_of_volumes_without_few_candidates(env, shape, kind):
    """few labels, smooth and evenly sloped volumes (most voxels hold nearly the
    maximum), and one whose only slope is in the last block"""
    torch, lib, runtime = env
    z, y, x = np.indices(shape)
    tri = lambda a: np.abs(a % 32 - 16) * 40
    v = {"labels": np.random.default_rng(3).integers(0, 8, size=shape), "more labels": np.random.default_rng(3).integers(0, 40, size=shape),
         "smooth": 3000 + 900 * np.sin(x / 30.0) + 900 * np.cos(y / 40.0 + z / 50.0), "slope": tri(x) + tri(y) + tri(z),
         "corner": 1000 + 3000 * ((x >= shape[2] - 2) & (y >= shape[1] - 2) & (z >= shape[0] - 2))}[kind].astype(np.uint16)
    sc = S.scene_tiny(film=(8, 8))
    sc.volume = v
    r = runtime.Renderer(sc, lib)
    try:
        gm = torch.zeros(shape, dtype=torch.int16, device="cuda")
        full = r.gradient_magnitude(gm.data_ptr())
        assert r.gradient_magnitude() == full
    finally:
        r.close()


@pytest.mark.parametrize("shape,brick", [((1, 1, 1), 1), ((2, 2, 2), 1), ((5, 3, 321), 1), ((5, 3, 322), 1), ((9, 7, 640), 2), ((4, 5, 641), 3),
                                         ((65, 66, 130), 64), ((129, 4, 129), 64), ((40, 33, 31), 5)])
def test_majorant_grid_ragged(env, oracle, shape, brick):
    """rows of one block and one more, odd and even rows, volumes of k bricks and one voxel"""
    torch, lib, _ = env
    rng = np.random.default_rng(brick)
    vol = rng.integers(0, 500, size=shape).astype(np.uint16)
    n = 500
    sig = np.abs(rng.normal(size=n)).astype(np.float32)
    sig[rng.random(n) < 0.5] = 0.0
    res = np.array(shape[::-1], dtype=np.int32)
    nb = [(d + brick - 1) // brick for d in shape]
    want = np.zeros(nb, dtype=np.float32)
    oracle.majorant_grid(OL.ptr(vol), OL.ptr(res), brick, OL.ptr(sig), n, 3.0, OL.ptr(want))
    d_vol, d_sig = torch.from_numpy(vol.view(np.int16)).cuda(), torch.from_numpy(sig).cuda()
    got = torch.zeros(nb, dtype=torch.float32, device="cuda")
    C.check(lib.er_build_majorant_device(d_vol.data_ptr(), res.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), brick, d_sig.data_ptr(), n, 3.0,
                                         got.data_ptr(), None))
    torch.cuda.synchronize()
    assert np.array_equal(bits(got.cpu().numpy()), bits(want))


@pytest.mark.parametrize("n", [1, 2, 4095, 4096, 4097, 5120, 16384, 65535, 65536])
def test_majorant_of_long_range_tables(env, oracle, n):
    """one block's table, tiles, and the levels behind the tiles'"""
    torch, lib, _ = env
    rng = np.random.default_rng(n)
    # bricks with ranges from one value to the whole table
    vol = np.minimum(rng.integers(0, n, size=(24, 20, 28)), (n - 1) * rng.random((24, 20, 28)) ** 6).astype(np.uint16)
    vol[8:16] = np.clip(n // 2 + rng.integers(-3, 4, size=vol[8:16].shape), 0, n - 1)
    sig = np.abs(rng.normal(size=n)).astype(np.float32)
    res = np.array(vol.shape[::-1], dtype=np.int32)
    nb = [(d + 3) // 4 for d in vol.shape]
    want = np.zeros(nb, dtype=np.float32)
    oracle.majorant_grid(OL.ptr(vol), OL.ptr(res), 4, OL.ptr(sig), n, 3.0, OL.ptr(want))
    d_vol, d_sig = torch.from_numpy(vol.view(np.int16)).cuda(), torch.from_numpy(sig).cuda()
    got = torch.zeros(nb, dtype=torch.float32, device="cuda")
    C.check(lib.er_build_majorant_device(d_vol.data_ptr(), res.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), 4, d_sig.data_ptr(), n, 3.0,
                                         got.data_ptr(), None))
    torch.cuda.synchronize()
    assert np.array_equal(bits(got.cpu().numpy()), bits(want))


@pytest.mark.parametrize("top", [900, 4095, 4096, 40000, 65535])
def test_march_map_of_long_tables(env, oracle, top):
    """volumes up to the largest voxel: opacity zero but for one band of values"""
    sc = S.scene_tiny(film=(24, 20), seed=3)
    rng = np.random.default_rng(top)
    v = (rng.random((22, 25, 27)) ** 8 * top).astype(np.uint16)
    v[10:13, 9:16, 9:20] = rng.integers(top * 3 // 4, top + 1, size=(3, 7, 11))
    v[11, 12, 13] = top
    sc.volume = v
    lo = 0.8 * top
    sc.tracer.opacity = C.make_plf([(0.0, 0.0), (lo, 0.0), (lo + 1.0, 0.6), (top + 1.0, 0.6)])
    check_sum(env, oracle, sc)


@pytest.mark.parametrize("w,h", [(1, 1), (63, 17), (64, 16), (65, 33), (3, 200)])
@pytest.mark.parametrize("radius", [0, 1, 5, 127])
def test_bilateral_tiles(env, oracle, w, h, radius):
    torch, lib, _ = env
    rng = np.random.default_rng(w + radius)
    img = rng.integers(0, 256, size=(h, w, 4), dtype=np.uint8)
    want, tmp = np.zeros_like(img), np.zeros_like(img)
    oracle.bilateral(OL.ptr(img), OL.ptr(tmp), OL.ptr(want), w, h, radius, 1.5, 20.0)
    d, t, o = torch.from_numpy(img).cuda(), torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda"), torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
    C.check(lib.er_bilateral_device(d.data_ptr(), t.data_ptr(), o.data_ptr(), w, h, radius, 1.5, 20.0, None))
    torch.cuda.synchronize()
    assert np.array_equal(t.cpu().numpy(), tmp) and np.array_equal(o.cpu().numpy(), want)


@pytest.mark.parametrize("w,h", [(65535 * 16 + 1, 1), (65535 * 16 + 20, 3), (2, 524280), (1030, 1001), (64 * 30, 16 * 20 - 1), (64 * 30 + 1, 16 * 20 - 1)])
def test_bilateral_of_large_images(env, oracle, w, h):
    """more columns than a grid has rows of tiles, as many rows as an image may
    have, and the last film of short tiles and the first of long ones"""
    torch, lib, _ = env
    img = np.random.default_rng(w).integers(0, 256, size=(h, w, 4), dtype=np.uint8)
    want, tmp = np.zeros_like(img), np.zeros_like(img)
    oracle.bilateral(OL.ptr(img), OL.ptr(tmp), OL.ptr(want), w, h, 2, 1.5, 20.0)
    d, t, o = torch.from_numpy(img).cuda(), torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda"), torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
    C.check(lib.er_bilateral_device(d.data_ptr(), t.data_ptr(), o.data_ptr(), w, h, 2, 1.5, 20.0, None))
    torch.cuda.synchronize()
    assert np.array_equal(t.cpu().numpy(), tmp) and np.array_equal(o.cpu().numpy(), want)


@pytest.mark.parametrize("stages", [0, 1])
@pytest.mark.parametrize("flags", [0, C.ER_BATCH_GRAPH])
def test_batch_windows_of_one_view(env, stages, flags):
    """views of over 2^20 samples in windows of their own beside views that
    share one, launched, advanced and launched again"""
    torch, lib, runtime = env
    sc = S.scene_tiny(res=24, film=(24, 20), seed=4)
    sc.tracer.settings.free_flight, sc.tracer.settings.mis, sc.tracer.settings.stratify = 1, 1, 1
    sc.tracer.settings.tune_stages = stages
    r = runtime.Renderer(sc, lib)
    rng = np.random.default_rng(3)
    sizes = [(24, 20, 3), (1025, 1024, 1), (33, 31, 2), (520, 512, 5), (16, 16, 3)]
    try:
        cams = [S.orbit_camera(rng, (w, h)) for w, h, _ in sizes]
        sums = [torch.zeros((h, w, 4), device="cuda") for w, h, _ in sizes]
        b = runtime.Batch([(r.tracer_id, spp, d.data_ptr(), cam) for (w, h, spp), d, cam in zip(sizes, sums, cams)], flags=flags)
        assert b.info()["windows"] > 1
        for first in (0, 7):
            if first:
                b.advance(first)
            b.launch()
            torch.cuda.synchronize()
            for i, ((w, h, spp), cam) in enumerate(zip(sizes, cams)):
                t = C.er_tracer_desc.from_buffer_copy(r.tracer_desc)
                t.camera = cam
                tid = ctypes.c_int32(-1)
                C.check(lib.er_bind_tracer(ctypes.byref(t), ctypes.byref(tid)))
                d = torch.zeros((h, w, 4), device="cuda")
                C.check(lib.er_trace_sum_device(tid.value, spp, i, first, d.data_ptr(), 0, None))
                torch.cuda.synchronize()
                lib.er_unbind_tracer(tid.value)
                assert torch.equal(d.view(torch.int32), sums[i].view(torch.int32)), (i, first)
        b.close()
    finally:
        r.close()


@pytest.mark.parametrize("stages", [0, 1])
@pytest.mark.parametrize("flags", [0, C.ER_BATCH_GRAPH])
def test_batch_of_full_windows(env, stages, flags):
    """two views that fill more than a window between them: each in windows of
    its own, its parameters by value, its first sample from the table"""
    torch, lib, runtime = env
    sc = S.scene_tiny(res=24, film=(24, 20), seed=4)
    s = sc.tracer.settings
    s.free_flight = s.mis = s.stratify = 1
    s.tune_stages, s.majorant_brick = stages, 2
    r = runtime.Renderer(sc, lib)
    rng = np.random.default_rng(5)
    try:
        cams = [S.orbit_camera(rng, (1025, 1024)) for _ in range(2)]
        sums = [torch.zeros((1024, 1025, 4), device="cuda") for _ in cams]
        b = runtime.Batch([(r.tracer_id, 5, d.data_ptr(), cam) for d, cam in zip(sums, cams)], flags=flags)
        assert b.info()["windows"] == b.info()["segments"] == 2
        for first in (0, 5):
            if first:
                b.advance(first)
            b.launch()
            torch.cuda.synchronize()
            for i, cam in enumerate(cams):
                t = C.er_tracer_desc.from_buffer_copy(r.tracer_desc)
                t.camera = cam
                tid = ctypes.c_int32(-1)
                C.check(lib.er_bind_tracer(ctypes.byref(t), ctypes.byref(tid)))
                d = torch.zeros((1024, 1025, 4), device="cuda")
                C.check(lib.er_trace_sum_device(tid.value, 5, i, first, d.data_ptr(), 0, None))
                torch.cuda.synchronize()
                lib.er_unbind_tracer(tid.value)
                assert torch.equal(d.view(torch.int32), sums[i].view(torch.int32)), (i, first)
        b.close()
    finally:
        r.close()
