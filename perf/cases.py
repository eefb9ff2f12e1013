"""What the renderer is measured on: the calls of its users, through the
package's public entry points (the runtime.Renderer, runtime.Batch and
medium.Medium classes and the C ABI behind them), from one small viewer frame
to batches over a gigabyte volume.

The scenes have the shapes, transfer functions, lights and cameras of the
workloads in the package's scenes module (c1: blobs and one area light; c2:
CT-like shells, 16-node transfer function, hybrid shading, three lights; c3
and c5: batches; c4: the differentiable medium), with volumes generated on
the GPU from the seed.

A case's `kind` says which calls it makes:

    frames       a viewer after a camera move: accumulation restarted, a few
                 frames of the reference's pipeline (RenderEstimate), RGBA8 read back
    frame        the same frame by the device-pointer entry points, for an
                 application that owns its buffers
    sum          many samples per pixel into a caller's sum buffer
    progressive  a viewer on the unbiased estimator: accumulation restarted,
                 a few short multi-sample renders, RGBA8 read back
    batch        many views in one submission
    medium       image of a differentiable medium and its gradients
    tf_edit      two edits of the opacity transfer function, each rendered and read back
    load         a new volume in an existing slot, rendered and read back
    display      post-processing of a film that the caller holds
"""
import ctypes
import importlib
import math

import numpy as np
import torch

PKG = importlib.import_module("exposure-render_gb300")
RUNTIME = importlib.import_module("exposure-render_gb300.runtime")
MEDIUM = importlib.import_module("exposure-render_gb300.medium")
C = PKG.capi
S = PKG.scenes


def listed():
    return [
        # a viewer window on a small data set with a floor and a ball beside
        # it: every event type of the reference; launches and latency count
        {"name": "frames_objects", "kind": "frames", "volume": "blobs", "rx": 96, "ry": 96, "rz": 96, "w": 320, "h": 240, "frames": 2,
         "objects": True},
        # the reference's frame on a CT-sized volume and a full window, its
        # post-processing and the bilateral filter on the caller's buffers
        {"name": "frame_ct", "kind": "frame", "volume": "shells", "rx": 512, "ry": 512, "rz": 512, "w": 1024, "h": 1024},
        # c1 as the reference estimates it: fixed-step march, phase function
        {"name": "sum_c1_march", "kind": "sum", "volume": "blobs", "rx": 128, "ry": 128, "rz": 128, "w": 256, "h": 256, "spp": 64,
         "delta": False, "shading": "phase", "brick": 8, "objects": False},
        # c2 on the unbiased estimator: delta tracking, hybrid shading, full MIS
        {"name": "sum_c2_delta", "kind": "sum", "volume": "shells", "rx": 512, "ry": 512, "rz": 512, "w": 1024, "h": 1024, "spp": 32,
         "delta": True, "shading": "hybrid", "brick": 4, "objects": False},
        # an interactive window of no round size on a cropped scan
        {"name": "progressive_odd", "kind": "progressive", "volume": "shells", "rx": 301, "ry": 257, "rz": 203, "w": 641, "h": 479,
         "passes": 2, "spp": 1, "brick": 4},
        # c3: a quarter of its views, films and samples over its three volumes
        {"name": "batch_c3", "kind": "batch", "scene": "c3", "views": 16, "film": 512, "spp": 128, "rx": 384, "ry": 384, "rz": 256,
         "brick": 2},
        # c5: large films of a gigabyte volume
        {"name": "batch_c5", "kind": "batch", "scene": "c5", "views": 2, "film": 2048, "spp": 16, "rx": 1024, "ry": 1024, "rz": 512,
         "brick": 4},
        # c4: image and gradients of the tracer's transport model
        {"name": "medium_tracer", "kind": "medium", "model": "tracer", "rx": 128, "ry": 128, "rz": 128, "w": 256, "h": 256, "spp": 32,
         "values": 64},
        # a small fit of the B-spline medium on an odd grid
        {"name": "medium_spline", "kind": "medium", "model": "spline", "rx": 72, "ry": 65, "rz": 81, "w": 150, "h": 111, "spp": 16,
         "values": 16},
        # the transfer-function editor over the CT-sized volume
        {"name": "tf_edit_ct", "kind": "tf_edit", "rx": 512, "ry": 512, "rz": 512, "w": 512, "h": 512, "brick": 4},
        # a time step of a volume sequence: new voxels, one picture
        {"name": "load_c3", "kind": "load", "rx": 384, "ry": 384, "rz": 256, "w": 512, "h": 512, "spp": 4, "brick": 2},
        # a 4K film tone-mapped and filtered for display
        {"name": "display_4k", "kind": "display", "w": 3840, "h": 2160, "radius": 2},
    ]


def _log(rng, lo, hi):
    """a whole number, spread evenly over the logarithm of [lo, hi]"""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("frames", "frame", "sum", "sum", "progressive", "batch", "medium", "medium", "tf_edit", "load", "display"))
    c = {"kind": kind}
    if kind in ("frames", "frame", "sum"):
        # the sides of the volume within a factor of two of each other
        c["volume"] = rng.choice(("blobs", "shells"))
        side = _log(rng, 48, 400)
        for a in ("rx", "ry", "rz"):
            c[a] = int(side * rng.uniform(0.7, 1.28))
        c["w"], c["h"] = _log(rng, 100, 1000), _log(rng, 100, 1000)
        if kind == "frames":
            c["frames"] = rng.randint(1, 3)
            c["objects"] = rng.random() < 0.5
        if kind == "sum":
            c["delta"] = rng.random() < 0.6
            c["shading"] = rng.choice(("brdf", "phase", "hybrid"))
            c["brick"] = rng.choice((1, 2, 3, 4, 8))
            c["objects"] = rng.random() < 0.3
            c["spp"] = max(1, min(_log(rng, 1, 128), (1 << 23) // (c["w"] * c["h"])))
    elif kind == "progressive":
        side = _log(rng, 48, 400)
        for a in ("rx", "ry", "rz"):
            c[a] = int(side * rng.uniform(0.7, 1.28))
        c.update(volume=rng.choice(("blobs", "shells")), w=_log(rng, 100, 1400), h=_log(rng, 100, 1400), passes=rng.randint(1, 4),
                 spp=rng.randint(1, 4), brick=rng.choice((2, 4, 8)))
    elif kind == "batch":
        c["scene"] = rng.choice(("c3", "c5"))
        side = _log(rng, 64, 400)
        for a in ("rx", "ry", "rz"):
            c[a] = int(side * rng.uniform(0.7, 1.28))
        c.update(views=rng.randint(2, 16), film=_log(rng, 100, 512), spp=_log(rng, 8, 128), brick=rng.choice((1, 2, 4, 8)))
    elif kind == "medium":
        side = _log(rng, 24, 128)
        for a in ("rx", "ry", "rz"):
            c[a] = int(side * rng.uniform(0.8, 1.0))
        c.update(model=rng.choice(("tracer", "spline")), w=_log(rng, 40, 256), h=_log(rng, 40, 256), spp=_log(rng, 2, 32),
                 values=rng.randint(8, 64))
    elif kind in ("tf_edit", "load"):
        side = _log(rng, 64, 400)
        for a in ("rx", "ry", "rz"):
            c[a] = int(side * rng.uniform(0.7, 1.28))
        c.update(w=_log(rng, 100, 800), h=_log(rng, 100, 800), brick=rng.choice((1, 2, 4, 8)))
        if kind == "load":
            c["spp"] = rng.randint(1, 8)
    else:
        c.update(w=_log(rng, 200, 3840), h=_log(rng, 200, 2160), radius=rng.randint(1, 5))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _host(volume):
    """the voxels in pinned host memory, as the bind calls take them"""
    out = torch.empty(volume.shape, dtype=torch.uint16, pin_memory=True)
    out.copy_(volume)
    return out.numpy()


def _axis(n):
    return torch.arange(n, device="cuda", dtype=torch.float32)


def _blob_sum(shape, rng, n, centre, sigma, amp):
    """a sum of n axis-aligned Gaussians on the grid, float32"""
    Z, Y, X = shape
    ext = np.array([X, Y, Z])
    v = torch.zeros(shape, device="cuda")
    for _ in range(n):
        m, s = rng.uniform(*centre, size=3) * ext, rng.uniform(*sigma, size=3) * ext
        gx, gy, gz = (torch.exp(-0.5 * ((_axis(k) - float(m[i])) / float(s[i])) ** 2) for i, k in enumerate((X, Y, Z)))
        v += (gz * float(rng.uniform(*amp)))[:, None, None] * (gy[:, None] * gx[None, :])
    return v


def _blobs(shape, seed):
    """twelve anisotropic blobs of amplitude 500 to 4000 over a noise floor"""
    v = _blob_sum(shape, np.random.default_rng(seed), 12, (0.2, 0.8), (0.04, 0.14), (500.0, 4000.0))
    v += 50.0 * torch.rand(shape, device="cuda", generator=_generator(seed))
    return _host(v.floor_().clamp_(0, 65535).to(torch.uint16))


def _shells(shape, seed):
    """nested shells in a soft-tissue ellipsoid, Gaussian noise inside it"""
    Z, Y, X = shape
    rng = np.random.default_rng(seed)
    a = rng.uniform(0.95, 1.05, size=3)
    L = float(max(shape))
    x, y, z = ((_axis(n) - (n - 1) / 2.0) / n for n in (X, Y, Z))
    ell = (z / float(0.36 * a[2])) ** 2
    ell = ell[:, None, None] + ((y / float(0.40 * a[1])) ** 2)[:, None] + ((x / float(0.46 * a[0])) ** 2)[None, :] <= 1.0
    m = min(shape) / L
    r2 = ((z * Z / L) ** 2)[:, None, None] + ((y * Y / L) ** 2)[:, None] + ((x * X / L) ** 2)[None, :]
    v = torch.where(ell, 1000.0, 0.0)
    for lo, hi, value in ((0.26, 0.30, 1400.0), (0.15, 0.19, 2500.0), (0.0, 0.07, 1400.0)):
        v = torch.where((r2 >= (lo * m) ** 2) & (r2 < (hi * m) ** 2), value, v)
    v += torch.where(ell, 30.0 * torch.randn(shape, device="cuda", generator=_generator(seed)), 0.0)
    return _host(v.floor_().clamp_(0, 65535).to(torch.uint16))


def _camera(rng, w, h):
    return S.orbit_camera(rng, (w, h), radius=float(rng.uniform(1.8, 2.4)))


SHADING = {"brdf": C.SHADING_BRDF_ONLY, "phase": C.SHADING_PHASE_ONLY, "hybrid": C.SHADING_HYBRID}


def _unbiased(t, brick):
    t.settings.free_flight = C.FREE_FLIGHT_DELTA
    t.settings.mis = C.MIS_FULL
    t.settings.stratify = 1
    t.settings.majorant_brick = brick


def _scene(case, seed, film):
    """the scene of a case's volume: blobs with the c1 tracer and light,
    shells with the c2 tracer and lights"""
    shape = (case["rz"], case["ry"], case["rx"])
    rng = np.random.default_rng(seed + 1)
    blobs = case.get("volume", "shells") == "blobs"
    volume = (_blobs if blobs else _shells)(shape, seed)
    lights, textures = S.c1_lights() if blobs else S.c2_lights()
    t = (S.c1_tracer if blobs else S.c2_tracer)(film)
    t.camera = _camera(rng, *film)
    t.settings.seed = 1 + seed % 65521
    sc = S.Scene("case", volume, tracer=t, lights=lights, textures=textures)
    if case.get("objects"):
        # the floor, the ball and their textures of the objects scene
        n = len(textures)
        sc.textures = textures + [S.uniform_texture((0.7, 0.5, 0.3)),
                                  S.checker_texture((0.3, 0.3, 0.3), (0.05, 0.05, 0.05), repeat=(4.0, 4.0)),
                                  S.uniform_texture((0.6, 0.6, 0.6))]
        floor = S.make_shape(C.SHAPE_PLANE, S.look_at_tm((0.0, 0.0, -0.6), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0)), size=(3.0, 3.0, 0.0))
        ball = S.make_shape(C.SHAPE_SPHERE, S.look_at_tm((0.55, -0.1, 0.25), (0.55, -0.1, 1.25), (0.0, 1.0, 0.0)), outer=0.2)
        sc.objects = [S.make_object(floor, n, n + 1, n + 2), S.make_object(ball, n, n, n + 2)]
        t.object_count = 2
        t.object_ids[0], t.object_ids[1] = 0, 1
    return sc


class State:
    """what a program holds; the library's slots are given back with it"""

    def __init__(self, case):
        self.case = case
        self.renderers, self.batch = [], None

    def bind(self, scene):
        r = RUNTIME.Renderer(scene)
        self.renderers.append(r)
        return r

    def __del__(self):
        if self.batch is not None:
            self.batch.close()
        for r in self.renderers:
            r.close()


def prepare(case, seed):
    seed = int(seed)
    s = State(case)
    kind = case["kind"]
    if kind in ("frames", "frame", "sum", "progressive"):
        sc = _scene(case, seed, (case["w"], case["h"]))
        t = sc.tracer
        if kind in ("frames", "frame"):
            # the reference's live path: BRDF at every event, light sampling
            t.settings.apply_shading_type = 0
            t.settings.mis = C.MIS_LIGHT_ONLY
            t.settings.bilateral = 0
        elif kind == "sum":
            t.settings.apply_shading_type = 0 if case["shading"] == "brdf" else 1
            t.settings.shading_type = SHADING[case["shading"]]
            if case["delta"]:
                _unbiased(t, case["brick"])
            else:
                t.settings.mis = C.MIS_LIGHT_ONLY
        else:
            _unbiased(t, case["brick"])
            t.settings.bilateral = 1
        s.r = s.bind(sc)
        n = case["w"] * case["h"]
        if kind == "frame":
            s.lanes = torch.randint(1, 2 ** 31 - 2, (2 * n,), device="cuda", dtype=torch.int32, generator=_generator(seed))
        elif kind == "sum":
            s.first = seed % 1000
    elif kind == "batch":
        _prepare_batch(s, case, seed)
    elif kind == "medium":
        _prepare_medium(s, case, seed)
    elif kind == "tf_edit":
        sc = _scene(case, seed, (case["w"], case["h"]))
        _unbiased(sc.tracer, case["brick"])
        s.r = s.bind(sc)
        # the editor moves the soft tissue's opacity back and forth
        o = sc.tracer.opacity
        nodes = [(float(o.position[i]), float(o.value[i])) for i in range(o.count)]
        s.opacities = [C.make_plf([(p, v * k if p < 1300.0 else v) for p, v in nodes]) for k in (0.0, 0.7 + 0.2 * (seed % 7) / 7)]
    elif kind == "load":
        case = dict(case, volume="blobs")
        sc = _scene(case, seed, (case["w"], case["h"]))
        _unbiased(sc.tracer, case["brick"])
        sc.tracer.settings.apply_shading_type = 1
        sc.tracer.settings.shading_type = C.SHADING_HYBRID
        s.r = s.bind(sc)
        s.desc = sc.volume_desc()
    else:
        g = _generator(seed)
        n = case["w"] * case["h"]
        s.film = torch.rand((case["h"], case["w"], 4), device="cuda", generator=g) * 1.5
        s.film[..., 3] = (s.film[..., 3] > 0.4).float()
        s.before = torch.rand((case["h"], case["w"], 4), device="cuda", generator=g)
        s.out = [torch.empty((n, 4), device="cuda", dtype=torch.uint8) for _ in range(3)]
    return s


def _prepare_batch(s, case, seed):
    rng = np.random.default_rng(seed)
    full = (case["rz"], case["ry"], case["rx"])
    if case["scene"] == "c3":
        # three volumes, the largest of them the case's
        shapes = [tuple(max(8, int(k * f)) for k in full) for f in (0.25, 0.64, 1.0)]
        volumes = [_blobs(shp, seed + k) for k, shp in enumerate(shapes)]
    else:
        volumes = [_shells(full, seed)]
    for v in volumes:
        if case["scene"] == "c3":
            lights, textures = S.c1_lights()
            t = S.c1_tracer((64, 64))
        else:
            lights, textures = S.c2_lights()
            t = S.c2_tracer((64, 64))
            t.settings.bilateral = 0
        _unbiased(t, case["brick"])
        t.settings.seed = 1 + seed % 65521
        if case["scene"] == "c3":
            t.settings.tune_stages = C.PERSISTENT_BOTH
        s.bind(S.Scene("case", v, tracer=t, lights=lights, textures=textures))
    views, s.sums = [], []
    # which volume, film and samples each view has is the same for every seed
    mix = np.random.default_rng(7)
    for _ in range(case["views"]):
        # films and samples per pixel of a quarter up to the case's own
        film, spp = case["film"], case["spp"]
        if case["scene"] == "c3":
            film, spp = max(16, film * int(mix.integers(1, 5)) // 4), int(mix.integers((spp + 3) // 4, spp + 1))
        d = torch.empty((film, film, 4), device="cuda")
        s.sums.append(d)
        r = s.renderers[int(mix.integers(0, len(volumes)))]
        views.append((r.tracer_id, spp, d.data_ptr(), _camera(rng, film, film)))
    s.batch = RUNTIME.Batch(views)


def _prepare_medium(s, case, seed):
    shape = (case["rz"], case["ry"], case["rx"])
    film = (case["w"], case["h"])
    rng = np.random.default_rng(seed)
    density = _blob_sum(shape, rng, 10, (0.25, 0.75), (0.06, 0.16), (0.3, 0.9)).clamp_(0.0, 1.0).contiguous()
    tracer = case["model"] == "tracer"
    # the tracer's volume only places the medium: its voxels are not read
    sc = (S.tf_medium_scene(res=shape, film=film, n_nodes=case["values"], emission=0.8) if tracer
          else S.medium_scene(res=shape, film=film))
    sc.tracer.camera = _camera(rng, *film)
    values = S.plf_node_values(sc.tracer.opacity) if tracer else S.ramp_opacity(case["values"])
    s.r = s.bind(sc)
    s.density = density.requires_grad_(True)
    s.opacity = torch.from_numpy(values).cuda().requires_grad_(True)
    with torch.no_grad():
        p = torch.nn.functional.pad(density[None, None], (1, 1, 1, 1, 1, 1), mode="replicate")[0, 0]
        g = [(p[1:-1, 1:-1, 2:] - p[1:-1, 1:-1, :-2]), (p[1:-1, 2:, 1:-1] - p[1:-1, :-2, 1:-1]), (p[2:, 1:-1, 1:-1] - p[:-2, 1:-1, 1:-1])]
        steepest = float(torch.sqrt(sum((k * 0.5 * max(shape)) ** 2 for k in g)).max())
    s.m = MEDIUM.Medium(s.r, s.density, s.opacity, 40.0, albedo=(0.8, 0.7, 0.6), model=case["model"],
                        gradient_magnitude_inv=1.0 / steepest if tracer else None)
    s.slope = torch.randn((case["h"], case["w"], 3), device="cuda", generator=_generator(seed)) / (case["w"] * case["h"])


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _reset(r):
    C.check(r.lib.er_reset_accumulation(r.tracer_id))


def run(s):
    c = s.case
    kind = c["kind"]
    if kind == "frames":
        _reset(s.r)
        for _ in range(c["frames"]):
            s.r.render_estimate()
        return s.r.get_estimate()
    if kind == "frame":
        w, h = c["w"], c["h"]
        lanes = s.lanes.clone()
        frame = torch.empty((h, w, 4), device="cuda")
        running = torch.zeros((h, w, 4), device="cuda")
        rgba, tmp, out = (torch.empty((h, w, 4), device="cuda", dtype=torch.uint8) for _ in range(3))
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        s.r.trace_frame_device(lanes.data_ptr(), frame.data_ptr(), stream)
        lib = s.r.lib
        C.check(lib.er_post_frame_device(frame.data_ptr(), running.data_ptr(), rgba.data_ptr(), w, h, 1, 1.0, 1, stream))
        C.check(lib.er_bilateral_device(rgba.data_ptr(), tmp.data_ptr(), out.data_ptr(), w, h, 2, 1.5, 20.0, stream))
        return {"lanes": lanes, "frame": frame, "running": running, "rgba": rgba, "filtered": out}
    if kind == "sum":
        out = torch.empty((c["h"], c["w"], 4), device="cuda")
        s.r.trace_sum_device(out.data_ptr(), c["spp"], 0, s.first, 0, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        return out
    if kind == "progressive":
        _reset(s.r)
        for _ in range(c["passes"]):
            s.r.render_spp(c["spp"])
        return s.r.get_estimate()
    if kind == "batch":
        s.batch.launch(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        return s.sums
    if kind == "medium":
        img = s.m(s.density, s.opacity, c["spp"])
        g_density, g_opacity = torch.autograd.grad(img, (s.density, s.opacity), s.slope)
        return {"image": img.detach(), "density": g_density, "opacity": g_opacity}
    if kind == "tf_edit":
        shots = []
        for o in s.opacities:
            s.r.tracer_desc.opacity = o
            s.r.rebind_tracer()
            _reset(s.r)
            s.r.render_spp(1)
            shots.append(s.r.get_estimate())
        return shots
    if kind == "load":
        vid = ctypes.c_int32(s.r.volume_id)
        C.check(s.r.lib.er_bind_volume(ctypes.byref(s.desc), ctypes.byref(vid)))
        _reset(s.r)
        s.r.render_spp(c["spp"])
        return s.r.get_estimate()
    # display
    w, h = c["w"], c["h"]
    lib = C.load_library()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    running = s.before.clone()
    rgba, tmp, out = s.out
    C.check(lib.er_post_frame_device(s.film.data_ptr(), running.data_ptr(), rgba.data_ptr(), w, h, 7, 1.0, 1, stream))
    C.check(lib.er_bilateral_device(rgba.data_ptr(), tmp.data_ptr(), out.data_ptr(), w, h, c["radius"], 1.5, 20.0, stream))
    return {"running": running, "rgba": rgba, "filtered": out}


# ---------------------------------------------------------------------------
# the least work, and 64-bit values
# ---------------------------------------------------------------------------

def work(case):
    """Bytes: the voxels (2 B, or 4 B with a gradient of 4 B) and the films
    once.  Operations: per sample some 500 (its seeds and camera ray, one
    event, its shading and the shadow segments' set-up), 8 per pixel and tap
    of the display filters, 600 per next-event estimate of the medium (about
    ten a sample, walked and shadowed once forward and once back)."""
    c = case
    kind = c["kind"]
    if kind == "display":
        n = c["w"] * c["h"]
        return {"bytes": n * (16 + 16 + 16 + 4 + 4), "flops": n * (9 * 8 + 4 * c["radius"] * 8)}
    voxels = c["rx"] * c["ry"] * c["rz"]
    if kind == "batch":
        f = (0.25 ** 3 + 0.64 ** 3 + 1.0) if c["scene"] == "c3" else 1.0
        # c3: the mean of a quarter to four quarters of the side, squared, and of the samples
        pix = c["views"] * c["film"] ** 2 * (0.469 if c["scene"] == "c3" else 1.0)
        samples = pix * c["spp"] * (0.625 if c["scene"] == "c3" else 1.0)
        return {"bytes": 2 * voxels * f + 16 * pix, "flops": 500 * samples}
    n = c["w"] * c["h"]
    if kind == "medium":
        return {"bytes": 8 * voxels + 24 * n, "flops": 12000 * n * c["spp"]}
    if kind == "frames":
        return {"bytes": 2 * voxels + 4 * n, "flops": 500 * n * c["frames"]}
    if kind == "frame":
        return {"bytes": 2 * voxels + n * (16 + 16 + 16 + 4 + 4), "flops": 500 * n}
    if kind == "sum":
        return {"bytes": 2 * voxels + 16 * n, "flops": 500 * n * c["spp"]}
    if kind == "progressive":
        return {"bytes": 2 * voxels + 4 * n, "flops": 500 * n * c["passes"] * c["spp"]}
    if kind == "tf_edit":
        return {"bytes": 2 * voxels + 8 * n, "flops": 1000 * n}
    return {"bytes": 2 * 2 * voxels + 4 * n, "flops": 500 * n * c["spp"]}


def exact(case, seed):
    """The display case's filtered running estimate: the 3x3 Gaussian of the
    film (alpha: the centre's over the weights' sum), and R += (F - R) / n.
    The other floating outputs are sums over random walks whose branches are
    taken on 32-bit values: a 64-bit evaluation takes other branches."""
    if case["kind"] != "display":
        return None
    s = prepare(case, seed)
    f, before = s.film.double(), s.before.double()
    h, w = f.shape[:2]
    acc = torch.zeros_like(f)
    tot = torch.zeros((h, w, 1), device="cuda", dtype=torch.float64)
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            k = math.exp(-(dx * dx + dy * dy) / 2.0)
            y0, y1, x0, x1 = max(0, -dy), min(h, h - dy), max(0, -dx), min(w, w - dx)
            acc[y0:y1, x0:x1] += k * f[y0 + dy:y1 + dy, x0 + dx:x1 + dx]
            tot[y0:y1, x0:x1] += k
    acc[..., 3] = f[..., 3]
    running = before + (acc / tot - before) / 7.0
    return {"running": running, "rgba": None, "filtered": None}
