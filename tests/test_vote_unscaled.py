"""The corner votes without the normalised line (voteUnscaled, beam_math.cuh):
wherever it gives an answer, the one that makeLine's float line gives, for
lines and corners over sixteen orders of magnitude, corners on the line, on
the band's edges and one or a few steps of the last bit beside them."""
import ctypes as C

import numpy as np
import pytest


@pytest.fixture(scope="module")
def vote():
    import build_emu
    lib = C.CDLL(build_emu.build())
    F = C.c_float

    def f(qx, qy, a, b, c, eps, ext):
        out = (C.c_int * 4)()
        known = lib.emu_vote((F * 4)(*qx), (F * 4)(*qy), F(a), F(b), F(c), F(eps), F(ext), out)
        return known, tuple(out)
    return f


@pytest.mark.parametrize("where", ["anywhere", "on the line", "on the band's edge"])
def test_agrees_with_the_line(where, vote):
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
            nn = np.hypot(float(a), float(b))
            for k in range(4):
                d = (qx[k] * float(a) + qy[k] * float(b) + float(c)) / nn
                w = 0.0 if where == "on the line" else eps * rng.choice([-1.0, 1.0])
                qx[k] += (w - d) * float(a) / nn
                qy[k] += (w - d) * float(b) / nn
        qx, qy = np.float32(qx), np.float32(qy)
        for k in range(4):
            for _ in range(rng.integers(0, 3)):
                qx[k] = np.nextafter(qx[k], np.float32(rng.choice([-1e30, 1e30])))
        known, out = vote(qx, qy, float(a), float(b), float(c), eps, ext)
        if known:
            told += 1
            assert out[:2] == out[2:], (qx, qy, a, b, c, ext)
    if where == "anywhere":
        assert told > 0.9 * n


@pytest.mark.parametrize("line", [(0, 0, 0), (0, 0, 1), (1e-30, 0, 1), (1, 0, 1e30), (np.nan, 1, 0), (1, np.inf, 0),
                                  (1e-40, 1e-40, 1e-40), (3e38, 3e38, 1)])
def test_leaves_odd_lines_to_the_caller(line, vote):
    assert not vote([0, 1, 1, 0], [0, 0, 1, 1], *line, 2e-5, 1.0)[0]
