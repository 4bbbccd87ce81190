"""The corner votes without the normalised line (voteUnscaled, beam_math.cuh):
wherever it gives an answer, the one that makeLine's float line gives, for
lines and corners over sixteen orders of magnitude, corners on the line, on
the band's edges and one or a few steps of the last bit beside them -- with the
norm as the host computes it, and off by as much as the device's approximate
root may be (the margin allows 2^-20 of it; rsqrtf and a product stay within
2.5 ulp, 2^-21.6 of it).  And over whole scenes, against the emulator's tests by
normalised lines."""
import ctypes as C

import numpy as np
import pytest


@pytest.fixture(scope="module")
def vote():
    import build_emu
    lib = C.CDLL(build_emu.build())
    F = C.c_float

    def f(qx, qy, a, b, c, eps, ext, off=0.0):
        out = (C.c_int * 4)()
        known = lib.emu_vote((F * 4)(*qx), (F * 4)(*qy), F(a), F(b), F(c), F(eps), F(ext), C.c_double(off), out)
        return known, tuple(out)
    return f


@pytest.mark.parametrize("off", [0.0, 0.99 * 2.0 ** -20, -0.99 * 2.0 ** -20], ids=["host", "norm above", "norm below"])
@pytest.mark.parametrize("where", ["anywhere", "on the line", "on the band's edge", "about the band's edge"])
def test_agrees_with_the_line(where, off, vote):
    rng = np.random.default_rng(11)
    told = 0
    n = 6000
    for _ in range(n):
        ext = float(np.float32(10.0 ** rng.uniform(-4, 4)))
        eps = float(np.float32(2e-5) * np.float32(ext))
        s = 10.0 ** rng.uniform(-8, 8)
        th = rng.uniform(0, 2 * np.pi)
        a, b = np.float32(s * np.cos(th)), np.float32(s * np.sin(th))
        c = np.float32(s * ext * rng.normal() * 10.0 ** rng.uniform(-3, 3))
        qx, qy = (rng.uniform(-1, 1, 4) * ext for _ in range(2))
        if where != "anywhere":  # moved along the normal to a wanted distance, then a few last bits off
            # (about the edge: from twice eps to a few last bits beside it; the margin is about a third of eps)
            nn = np.hypot(float(a), float(b))
            for k in range(4):
                d = (qx[k] * float(a) + qy[k] * float(b) + float(c)) / nn
                w = 0.0 if where == "on the line" else eps * rng.choice([-1.0, 1.0])
                if where.startswith("about"):
                    w *= 1 + rng.choice([-1.0, 1.0]) * 2.0 ** rng.uniform(-12, 1)
                qx[k] += (w - d) * float(a) / nn
                qy[k] += (w - d) * float(b) / nn
        qx, qy = np.float32(qx), np.float32(qy)
        for k in range(4):
            for _ in range(rng.integers(0, 3)):
                qx[k] = np.nextafter(qx[k], np.float32(rng.choice([-1e30, 1e30])))
        known, out = vote(qx, qy, float(a), float(b), float(c), eps, ext, off)
        if known:
            told += 1
            assert out[:2] == out[2:], (qx, qy, a, b, c, ext)
    # It has to answer away from the edges, where only a |c| far above the extent
    # (a third of the lines here) makes the margin wider than eps, and never on one.
    least, most = {"anywhere": (0.9, 1), "on the line": (0.5, 1), "on the band's edge": (0, 0.01),
                   "about the band's edge": (0.05, 0.5)}[where]
    assert least * n <= told <= most * n


@pytest.mark.parametrize("line", [(0, 0, 0), (0, 0, 1), (1e-30, 0, 1), (1, 0, 1e30), (np.nan, 1, 0), (1, np.inf, 0),
                                  (1e-40, 1e-40, 1e-40), (3e38, 3e38, 1)])
def test_leaves_odd_lines_to_the_caller(line, vote):
    assert not vote([0, 1, 1, 0], [0, 0, 1, 1], *line, 2e-5, 1.0)[0]


@pytest.mark.parametrize("name", ["room", "plant", "displaced_sphere"])
def test_scenes_by_the_line(name, native_lib):
    from conftest import scene
    from beamtrace2007_b200.renderer import make_camera
    from emu import Emulator
    s, ps = scene(name, **({"subdiv": 4} if name == "displaced_sphere" else {}))
    em = Emulator(ps)
    v = s.views[0]
    cam = make_camera(v.eye, v.target, v.fov, s.up, 33, 27)
    before = em.tests()
    pe, _ = em.primary_tiles(cam, tile=8)
    em.point(cam, np.array(s.point_light, np.float32), pe.select(pe.tri >= 0))
    tri = np.arange(0, ps.num_tris, max(1, ps.num_tris // 150), dtype=np.int32)
    light = s.light_array(1.5)
    X = ps.pos[ps.tris[tri].astype(np.int64)].mean(1).astype(np.float32)
    N = ps.tri_normals[tri]
    N = np.where((N * (light[:3] - X)).sum(1, keepdims=True) < 0, -N, N).astype(np.float32)
    em.soft_points(light.astype(np.float32), ps.offset, tri, X, N, exact=True)
    run, differ = (a - b for a, b in zip(em.tests(), before))
    assert run > 10000 and differ == 0
