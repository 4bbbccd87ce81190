"""The lane-group kernels (csrc/group_core.cuh) against the host emulator of
the one-lane steps (tests/native/emu.cpp): the same pieces bit for bit and the
same counters, over meshes whose clips give triangles, quads, pentagons and
slivers, with rounds forced into full or tail kernels."""
import numpy as np
import pytest

from conftest import piece_keys, scene

pytestmark = pytest.mark.gpu

COUNTERS = ["kd_steps", "leaf_visits", "tri_tests", "hits", "splits", "beams", "root_beams", "presplit_beams",
            "five_splits", "climbs"]
# never tail rounds, no record handed on early; tail rounds throughout; tail rounds that leave a queue grown past
# 2 x 300 records to full rounds; full rounds with records handed on early; the default
MODES = {"full": dict(tail_records=-1, yield_pct=-1), "tail": dict(tail_records=1 << 30),
         "tail then full": dict(tail_records=300), "yield": dict(tail_records=-1, yield_pct=1), "default": {}}


def _soup(n=300, seed=5):
    """Random interpenetrating triangles."""
    from beamtrace2007_b200.renderer import PreparedScene
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1, 1, (n, 1, 3))
    pos = (c + rng.normal(0, 0.35, (n, 3, 3))).reshape(-1, 3).astype(np.float32)
    return PreparedScene(pos, np.arange(3 * n, dtype=np.uint32).reshape(-1, 3))


def _setup(name):
    from beamtrace2007_b200.renderer import make_camera
    if name == "soup":
        ps = _soup()
        return ps, make_camera((2.2, 1.1, 2.6), (0, 0, 0), 55.0, (0, 1, 0), 45, 37), (0.3, 3.0, 0.2), \
            np.array([0.3, 3.0, 0.2, 0.9, 0, 0, 0, 0, 0.9])
    s, ps = scene(name, **({"subdiv": 4} if name == "displaced_sphere" else {}))
    v = s.views[0]
    return ps, make_camera(v.eye, v.target, v.fov, s.up, 45, 37), s.point_light, s.light_array(1.5)


def _took_its_path(mode, info):
    """Whether a pass of at most 8192 roots went the way its mode is named after."""
    tails, others, yields = info["tail_rounds"], info["rounds"] - info["tail_rounds"], info["yields"]
    return {"full": tails == 0 and yields == 0, "tail": tails > 0 and others == 0,
            "tail then full": tails > 0 and others > 0 and info["max_spill"] > 600,
            "yield": tails == 0 and yields > 0, "default": tails > 0}[mode]


def _counters(info, st):
    return {k: (info[k], int(st[i])) for i, k in enumerate(COUNTERS) if info[k] != int(st[i])}


@pytest.mark.parametrize("name", ["room", "plant", "displaced_sphere", "soup"])
@pytest.mark.parametrize("mode", MODES)
def test_pieces_and_counters_equal_emulator(name, mode, gpu):
    from beamtrace2007_b200.renderer import GpuRenderer
    from emu import Emulator
    ps, cam, point, light = _setup(name)
    em = Emulator(ps)
    light_f = light.astype(np.float32)
    with GpuRenderer(ps, budget=1 << 20, primary_budget=1 << 20, **MODES[mode]) as g:
        for tile in (3, 16):
            prim = g.primary(cam, tile=tile)
            info = g.last_info
            pe, st = em.primary_tiles(cam, tile=tile)
            assert np.array_equal(piece_keys(prim, True), piece_keys(pe.select(pe.tri >= 0), True))
            assert info["retried_roots"] == 0 and _counters(info, st) == {}
            assert _took_its_path(mode, info) or (mode == "tail then full" and tile == 16)  # (nine roots: may stay small)
            assert abs(info["dropped_area"] - float(st[10:11].view(np.float64)[0])) <= 1e-9
        sh = g.point_shadows(cam, prim, point)
        info = g.last_info
        pe, st = em.point(cam, point, prim)
        assert np.array_equal(piece_keys(sh), piece_keys(pe))
        assert info["retried_roots"] == 0 and _counters(info, st) == {}
        # shading points: the mean of each visible polygon's triangle corners, lifted to its plane
        tri = prim.tri[:: max(1, len(prim) // 300)]
        corners = ps.pos[ps.tris[tri].astype(np.int64)].astype(np.float64)
        X = corners.mean(1).astype(np.float32)
        N = ps.tri_normals[tri]
        N = np.where((N.astype(np.float64) * (light[:3] - X)).sum(1, keepdims=True) < 0, -N, N).astype(np.float32)
        r = g.soft_points(light, tri, X, N, exact=True, offset=ps.offset)
        vis, G, st = em.soft_points(light_f, ps.offset, tri, X, N, exact=True)
        assert r.info["retried_roots"] == 0 and _counters(r.info, st) == {}
        # fixed point against double sums of the same pieces, each rounded to float
        assert np.abs(r.vis - vis).max() <= 1e-6 and np.abs(r.E - G).max() <= 1e-6 * max(1.0, np.abs(G).max())


@pytest.mark.parametrize("fov, tile", [(179.995, 16), (179.998, 16), (179.9999, 4), (179.9999, 16)])
def test_views_close_to_180_degrees(fov, tile, gpu):
    """A root's eps is 2e-5 of its extent on the image plane and passes 1 at an
    extent of 5e4: a record without a hit has no depth line to be outside of."""
    from beamtrace2007_b200.renderer import GpuRenderer, make_camera
    from emu import Emulator
    s, ps = scene("room")
    v = s.views[0]
    cam = make_camera(v.eye, v.target, fov, s.up, 16, 16)
    pe, st = Emulator(ps).primary_tiles(cam, tile=tile)
    pe = pe.select(pe.tri >= 0)
    assert len(pe) > 0
    for mode in (dict(tail_records=-1), {}):
        with GpuRenderer(ps, **mode) as g:
            prim = g.primary(cam, tile=tile)
            assert np.array_equal(piece_keys(prim, True), piece_keys(pe, True))
            assert _counters(g.last_info, st) == {}


@pytest.mark.parametrize("name, size, tile, capacity", [("plant", (45, 33), 16, 5120), ("plant", (45, 33), 16, 6656),
                                                        ("meeting", (64, 48), 8, 7168)])
def test_queues_near_their_capacity(name, size, tile, capacity, gpu):
    """Roots that need about all of a small queue: the pass ends with every
    piece, or with roots still over budget after the last retry -- never with a
    queue that holds more records than were reserved for."""
    from beamtrace2007_b200 import _native
    from beamtrace2007_b200.renderer import GpuRenderer, make_camera
    from emu import Emulator
    s, ps = scene(name)
    v = s.views[0]
    cam = make_camera(v.eye, v.target, v.fov, s.up, *size)
    pe, _ = Emulator(ps).primary_tiles(cam, tile=tile)
    want = piece_keys(pe.select(pe.tri >= 0), True)
    for _ in range(3):
        with GpuRenderer(ps, primary_budget=256, capacity=capacity) as g:
            try:
                prim = g.primary(cam, tile=tile)
            except _native.BtError as e:
                assert "still over budget" in str(e)
                continue
            assert g.last_info["max_spill"] <= capacity
            assert np.array_equal(piece_keys(prim, True), want)


def test_retried_root_fits_in_full_rounds(gpu):
    """One root that a queue holds in full rounds but not with every chain of
    splits run to its end at once: the retry passes have to find it room."""
    from beamtrace2007_b200.renderer import GpuRenderer, make_camera
    from emu import Emulator
    s, ps = scene("displaced_sphere", subdiv=5)
    v = s.views[0]
    cam = make_camera(v.eye, v.target, v.fov, s.up, 45, 33)
    pe, _ = Emulator(ps).primary_tiles(cam, tile=45)
    with GpuRenderer(ps, capacity=12288) as g:
        prim = g.primary(cam, tile=45)
        assert g.last_info["retried_roots"] > 0
    assert np.array_equal(piece_keys(prim, True), piece_keys(pe.select(pe.tri >= 0), True))


@pytest.mark.parametrize("name", ["room", "plant", "displaced_sphere", "soup"])
@pytest.mark.parametrize("tail_records", [-1, 1 << 30], ids=["full", "tail"])
def test_abandoned_roots(name, tail_records, gpu):
    """Budgets that most splitting roots outgrow: records of abandoned roots meet
    the clip and tail kernels at every place, and their roots come out of the
    retries whole (the counters hold the abandoned attempts too)."""
    from beamtrace2007_b200.renderer import GpuRenderer
    from emu import Emulator
    ps, cam, point, light = _setup(name)
    em = Emulator(ps)
    with GpuRenderer(ps, budget=4, primary_budget=8, tail_records=tail_records) as g:
        for tile in (3, 16):
            prim = g.primary(cam, tile=tile)
            info = g.last_info
            pe, st = em.primary_tiles(cam, tile=tile)
            assert np.array_equal(piece_keys(prim, True), piece_keys(pe.select(pe.tri >= 0), True))
            assert 0 < info["overflow_roots"] <= info["retried_roots"] and info["passes"] > 1
            assert (info["tail_rounds"] == 0) == (tail_records < 0)
            assert [k for i, k in enumerate(COUNTERS) if info[k] < int(st[i])] == []
        sh = g.point_shadows(cam, prim, point)
        pe, _ = em.point(cam, point, prim)
        assert np.array_equal(piece_keys(sh), piece_keys(pe))


@pytest.mark.parametrize("tail_records", [(1 << 30) - 1, 1 << 30, 1 << 62, (1 << 63) - 1])
def test_huge_tail_records(tail_records, gpu):
    """Any large tail_records means tail rounds always: twice the value may not
    fit the kernels' int, nor an int64."""
    from beamtrace2007_b200.renderer import GpuRenderer
    from emu import Emulator
    ps, cam, _, _ = _setup("room")
    pe, st = Emulator(ps).primary_tiles(cam, tile=16)
    with GpuRenderer(ps, tail_records=tail_records) as g:
        prim = g.primary(cam, tile=16)
        assert np.array_equal(piece_keys(prim, True), piece_keys(pe.select(pe.tri >= 0), True))
        assert _counters(g.last_info, st) == {} and g.last_info["tail_rounds"] == g.last_info["rounds"] > 0


def test_retries_of_a_large_budget(gpu):
    """16 times a budget of 2^20, four times over, is past an int."""
    from beamtrace2007_b200.renderer import GpuRenderer, make_camera
    from emu import Emulator
    s, ps = scene("plant")
    v = s.views[0]
    cam = make_camera(v.eye, v.target, v.fov, s.up, 45, 33)
    pe, _ = Emulator(ps).primary_tiles(cam, tile=3)
    with GpuRenderer(ps, primary_budget=1 << 20, capacity=4096) as g:
        prim = g.primary(cam, tile=3)
        assert g.last_info["passes"] > 3
    assert np.array_equal(piece_keys(prim, True), piece_keys(pe.select(pe.tri >= 0), True))
