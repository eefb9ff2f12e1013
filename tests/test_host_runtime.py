"""The library's host code on a machine without a GPU: its objects linked
against fake_cudart.cpp, which makes copies on the host and lists launches,
copies and waits by stream."""
import ctypes
import importlib
import os
import subprocess

import numpy as np
import pytest

import oracle_lib as OL

C = OL.C
S = OL.PKG.scenes
BUILD = importlib.import_module("exposure-render_gb300.build")
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def fake_path(tmp_path_factory):
    BUILD.build()
    out = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    objs = [os.path.join(BUILD.OUT, os.path.splitext(u)[0] + ".o") for u in BUILD.UNITS]
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(BUILD.nvcc()))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic,--no-undefined", "-I" + cuda,
                    os.path.join(HERE, "fake_cudart.cpp"), *objs, "-o", out], check=True)
    return out


@pytest.fixture()
def lib(fake_path, monkeypatch, tmp_path):
    monkeypatch.setenv("ER_TUNE_CACHE", str(tmp_path / "autotune.txt"))
    L = C.load_library(fake_path)
    L.fake_log.restype = ctypes.c_char_p
    L.fake_bad_read.argtypes = L.fake_largest_allocation.argtypes = [ctypes.c_size_t]
    L.fake_no_memory(0)
    L.fake_bad_read(0)
    L.fake_clear()
    yield L
    L.fake_jobs_each(0)
    L.fake_largest_allocation(ctypes.c_size_t(-1).value)
    L.fake_no_memory(0)
    L.fake_bad_read(0)
    L.er_reset()


def log(lib):
    """(what, stream, kernel or event) of every call since the last look"""
    out = [tuple(line.split(" ", 2)) for line in lib.fake_log().decode().splitlines()]
    lib.fake_clear()
    return out


def renderer(lib, sc):
    return importlib.import_module("exposure-render_gb300.runtime").Renderer(sc, lib)


STREAM_A, STREAM_B = 0x1000, 0x2000


def medium_desc(p):
    m = C.er_medium_desc()
    m.d_density, m.d_opacity, m.n_opacity, m.scale, m.nee_probability = p, p, 16, 1.0, 0.5
    m.d_majorant, m.brick, m.model = p, 8, C.ER_MEDIUM_SPLINE
    return m


@pytest.mark.parametrize("back", [False, True], ids=["forward", "adjoint"])
def test_medium_calls_on_two_streams_take_turns(lib, back):
    """the walks of one device share their job and item arrays: a call on
    another stream starts behind the work of the call before it"""
    sc = S.medium_scene(res=(8, 8, 8), film=(8, 8))
    r = renderer(lib, sc)
    buf = np.zeros(1 << 16, np.float32)
    p = buf.ctypes.data
    m = medium_desc(p)

    def call(stream):
        if back:
            C.check(lib.er_medium_adjoint(r.tracer_id, ctypes.byref(m), 2, 0, 0, p, None, p, p, stream))
        else:
            C.check(lib.er_medium_render(r.tracer_id, ctypes.byref(m), 2, 0, 0, p, p, stream))

    call(STREAM_A)
    first = log(lib)
    call(STREAM_B)
    second = log(lib)
    r.close()
    a, b = f"{STREAM_A:x}", f"{STREAM_B:x}"
    work = [i for i, e in enumerate(first) if e[0] in ("launch", "set") and e[1] == a and "k_dm_reduce" not in e[2]]
    marks = [(i, e[2]) for i, e in enumerate(first) if e[0] == "record" and e[1] == a]
    assert marks and marks[-1][0] > work[-1]
    begin = next(i for i, e in enumerate(second) if e[0] in ("launch", "set") and e[1] == b)
    assert ("wait", b, marks[-1][1]) in second[:begin]


def batch_info(lib, r, sizes, cap=0):
    """(windows, segments) of a batch of (width, height, samples) views"""
    runtime = importlib.import_module("exposure-render_gb300.runtime")
    rng = np.random.default_rng(1)
    views = [(r.tracer_id, spp, 0x100000 * (i + 1), S.orbit_camera(rng, (w, h))) for i, (w, h, spp) in enumerate(sizes)]
    b = runtime.Batch(views, flags=0, window_items=cap, lib=lib)
    info = b.info()
    b.close()
    return info["windows"], info["segments"]


@pytest.mark.parametrize("sizes,cap,want", [
    ([(200, 200, 16)] * 8, 0, (1, 8)),                              # 5.1 M samples: one window, however many views
    ([(1024, 1024, 1)] * 8, 0, (1, 8)),
    ([(1920, 1080, 1)] * 4, 0, (1, 4)),
    ([(1024, 1024, 5)] * 2, 0, (2, 2)),                             # two windows in any case: one view each
    ([(30, 20, 3), (30, 20, 3), (30, 20, 4)], 6000, (1, 3)),
    ([(30, 20, 6), (30, 20, 6), (30, 20, 6)], 6000, (2, 4)),        # 10800 samples: the second view in both
    ([(30, 20, 10), (30, 20, 10)], 6000, (2, 2)),
    ([(30, 20, 9), (30, 20, 2), (30, 20, 10)], 6000, (3, 3)),
    ([(30, 20, 25)], 6000, (3, 3)),
    ([(1100, 1000, 1), (20, 20, 1)], 0, (2, 2)),                    # the reduce stage's grid is the larger film's
])
def test_windows_are_as_few_as_can_be(lib, sizes, cap, want):
    """each window ends with its longest rays alone on the chip, so a view gets
    a window of its own only where that adds none"""
    sc = S.scene_tiny(res=8, film=(8, 8))
    sc.tracer.settings.free_flight = C.FREE_FLIGHT_DELTA
    r = renderer(lib, sc)
    try:
        assert batch_info(lib, r, sizes, cap) == want
    finally:
        r.close()


@pytest.mark.parametrize("side,spp,steps", [(64, 1, True), (512, 9, True), (1024, 2, True), (512, 10, False), (1024, 8, False)])
def test_shadow_stage_of_a_small_window_runs_in_steps(lib, side, spp, steps):
    """up to 16 samples for each lane of the resident wave (152 SMs of 1024)"""
    sc = S.scene_tiny(res=8, film=(side, side))
    sc.tracer.settings.free_flight = C.FREE_FLIGHT_DELTA
    r = renderer(lib, sc)
    d = np.zeros((side, side, 4), np.float32)
    log(lib)
    r.trace_sum_device(d.ctypes.data, spp)
    names = [e[2] for e in log(lib) if "k_wf_shadow_pt" in e[2]]
    r.close()
    assert len(names) == 1 and ("Lb1ELb0ELb1E" if steps else "Lb1ELb0ELb0E") in names[0]


def edit(lib, r, box, value):
    off, size = (ctypes.c_int32 * 3)(*box[0]), (ctypes.c_int32 * 3)(*box[1])
    v = np.full(box[1][::-1], value, np.uint16)
    return lib.er_update_volume_region(r.volume_id, off, size, v.ctypes.data)


def tune_key(lib, r, path):
    """the key under which the autotuner stores its choice"""
    r.autotune(1)
    with open(path) as f:
        return f.read().split()[-7]


BOXES = [((0, 0, 0), (30, 4, 4)), ((5, 6, 7), (20, 11, 3)), ((3, 6, 7), (20, 11, 9))]


@pytest.mark.parametrize("memory", [True, False], ids=["room", "no-room"])
def test_tuning_key_made_late_equals_one_made_at_once(lib, monkeypatch, tmp_path, memory):
    """a bind and its edits give the key that they give when the key is made
    after the bind, also when the device has no room for what the key needs"""
    keys = []
    for late in (False, True):
        path = tmp_path / f"{late}.txt"
        monkeypatch.setenv("ER_TUNE_CACHE", str(path))
        sc = S.scene_tiny(res=32, film=(8, 8), seed=5)
        r = renderer(lib, sc)
        if not late:
            tune_key(lib, r, path)
        lib.fake_no_memory(0 if memory else 1)
        for i, box in enumerate(BOXES):
            C.check(edit(lib, r, box, 100 + i))
        lib.fake_no_memory(0)
        keys.append(tune_key(lib, r, path))
        r.close()
    assert keys[0] == keys[1]


@pytest.mark.parametrize("memory", [True, False], ids=["room", "no-room"])
def test_tuning_key_of_a_volume_bound_again(lib, monkeypatch, tmp_path, memory):
    """an ID that held another, edited volume gives the new one's key"""
    keys = []
    for again in (False, True):
        path = tmp_path / f"{again}.txt"
        monkeypatch.setenv("ER_TUNE_CACHE", str(path))
        sc = S.scene_tiny(res=32, film=(8, 8), seed=5)
        r = renderer(lib, sc)
        lib.fake_no_memory(0 if memory else 1)
        if again:
            C.check(edit(lib, r, BOXES[1], 77))
            vd, vid = sc.volume_desc(), ctypes.c_int32(r.volume_id)
            C.check(lib.er_bind_volume(ctypes.byref(vd), ctypes.byref(vid)))
        C.check(edit(lib, r, BOXES[0], 100))
        lib.fake_no_memory(0)
        keys.append(tune_key(lib, r, path))
        r.close()
    assert keys[0] == keys[1]


def test_an_edit_stands_when_its_key_cannot_be_made(lib):
    """edits whose log is over a megabyte make the key: a failure there leaves
    the edit made, and the next render with its tables"""
    n = 256
    sc = S.scene_tiny(res=8, film=(8, 8))
    sc.volume = np.zeros((n, n, n), np.uint16)
    r = renderer(lib, sc)
    d = np.zeros((8, 8, 4), np.float32)
    r.trace_sum_device(d.ctypes.data, 1)
    lib.fake_bad_read((n ** 3 + 60) // 61 * 2)
    for i in range(2):
        assert edit(lib, r, ((0, 0, 0), (n, n, n)), i) == C.ER_OK
        log(lib)
        r.trace_sum_device(d.ctypes.data, 1)
        assert any("k_sigma_table" in e[2] for e in log(lib) if e[0] == "launch")
    r.close()


def fnv1a(h, b):
    for x in bytes(b):
        h = ((h ^ x) * 1099511628211) % (1 << 64)
    return h


def test_choices_timed_on_other_kernels_are_not_taken(lib, tmp_path):
    """a cache line under the key without the kernels' number (device, volume,
    settings) is not applied"""
    sc = S.scene_tiny(res=16, film=(8, 8), seed=5)
    r = renderer(lib, sc)
    t = r.tracer_desc
    s = C.er_render_settings.from_buffer_copy(t.settings)
    for f in ("majorant_brick", "tune_primary", "tune_shadow", "tune_shade", "tune_stages", "seed", "bilateral", "bilateral_radius", "frame_filter"):
        setattr(s, f, 0)
    s.bilateral_sigma_d = s.bilateral_sigma_r = 0.0
    i32 = lambda *v: np.array(v, np.int32).tobytes()
    volume = fnv1a(fnv1a(14695981039346656037, i32(16, 16, 16)), sc.volume.ravel()[::61].astype(np.uint16).tobytes())
    h = fnv1a(14695981039346656037, b"no GPU" + i32(152) + volume.to_bytes(8, "little") + np.array(sc.spacing, np.float32).tobytes())
    h = fnv1a(h, bytes(s) + bytes(t.opacity) + bytes(t.glossiness) + i32(t.camera.film_size[0], t.camera.film_size[1], t.light_count, 1))
    (tmp_path / "autotune.txt").write_text(f"{h:016x} 8 2 2 2 1.000 0\n")
    assert not r.autotune(1)["from_cache"]
    assert r.autotune(1)["from_cache"]
    r.close()


@pytest.mark.parametrize("tune", [2, 3, 4, 6, 8])
@pytest.mark.parametrize("mix", ["march", "delta", "both"])
def test_batch_tuning_picks_the_kernels(lib, mix, tune):
    """er_batch_set_tuning names the occupancy of the tracking stages in every
    batch; 8 is a variant of the batches that march"""
    runtime = importlib.import_module("exposure-render_gb300.runtime")
    kinds = {"march": (0, 0), "delta": (1, 1), "both": (0, 1)}[mix]
    rs = []
    for k in kinds:
        sc = S.scene_tiny(res=8, film=(8, 8))
        sc.tracer.settings.free_flight = k
        sc.tracer.settings.tune_stages = C.PERSISTENT_NONE
        rs.append(renderer(lib, sc))
    b = runtime.Batch([(r.tracer_id, 2, 0x100000 * (i + 1), None) for i, r in enumerate(rs)], flags=0, lib=lib)
    b.set_tuning(tune, tune)
    log(lib)
    b.launch()
    names = [e[2] for e in log(lib) if e[0] == "launch"]
    want = 4 if mix == "delta" and tune == 8 else tune
    for stage in ("k_wf_primary", "k_wf_shadow"):
        assert [n.split("ILi")[1].split("E")[0] for n in names if stage + "I" in n] == [str(want)], names
    b.close()
    for r in rs:
        r.close()


def test_gradient_maximum_of_small_values_goes_one_way(lib):
    """a volume whose values are within the bounds' error makes the full pass alone"""
    r = renderer(lib, S.scene_tiny(res=16, film=(8, 8)))
    log(lib)
    r.gradient_magnitude()
    assert len([e for e in log(lib) if e[0] == "launch"]) == 1
    r.close()


@pytest.mark.parametrize("n,blocks_of_one", [(300, True), (4096, True), (4097, False), (65536, False)])
def test_long_range_tables_are_not_one_blocks_work(lib, n, blocks_of_one):
    buf = np.zeros(1 << 21, np.float32)
    res = (ctypes.c_int32 * 3)(8, 8, 8)
    log(lib)
    C.check(lib.er_build_majorant_device(buf.ctypes.data, res, 8, buf.ctypes.data, n, 1.0, buf.ctypes.data, None))
    names = [e[2] for e in log(lib) if "k_rmq" in e[2]]
    assert any("k_rmqPK" in x for x in names) == blocks_of_one


def test_medium_without_room_for_its_jobs_takes_smaller_windows(lib):
    """the estimates of all samples get job slots, also those that find no light
    sample: a window whose jobs do not fit is walked in halves"""
    sc = S.medium_scene(res=(8, 8, 8), film=(32, 32))
    r = renderer(lib, sc)
    buf = np.zeros(1 << 18, np.float32)
    m = medium_desc(buf.ctypes.data)
    lib.fake_jobs_each(100)
    # the items' arrays fit; 64 samples of 1024 pixels have 100 MiB of points, 16 have 25
    lib.fake_largest_allocation((1 << 21) * 16)
    C.check(lib.er_medium_render(r.tracer_id, ctypes.byref(m), 64, 0, 0, buf.ctypes.data, buf.ctypes.data, None))
    assert sum("k_dm_gather" in e[2] for e in log(lib) if e[0] == "launch") == 4
    r.close()
