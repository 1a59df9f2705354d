"""The sphere roots in pairs of FP32 numbers (sphere_root_pair, csrc/sphere_pair.h) against
the FP64 test that stands behind them: wherever the pairs decide, miss or hit, the rounded
root and the side of the unrounded one are FP64's, bit for bit; and in scenes of ordinary
size they decide nearly always.  No GPU."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from chakumrender_gb300 import ckr

N = 300000


def unit(v):
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def roots(rows, mode):
    f = ckr.lib().ckr_internal_sphere_roots_host
    f.argtypes, f.restype = [C.c_void_p, C.c_uint32, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p], C.c_int
    rows = np.ascontiguousarray(rows, np.float32)
    n = len(rows)
    t, rem, code = np.empty(n, np.float32), np.empty(n, np.float32), np.empty(n, np.int32)
    assert f(rows.ctypes.data, n, mode, t.ctypes.data, rem.ctypes.data, code.ctypes.data) == 0
    return t, rem, code


def case(name):
    rng = np.random.default_rng(11)
    c, r = rng.uniform(-1, 1, (N, 3)), rng.uniform(0.05, 0.5, N)
    o, d = rng.uniform(-2, 2, (N, 3)), unit(rng.normal(size=(N, 3)))
    tmin = np.where(rng.random(N) < 0.2, rng.uniform(0, 2, N), 0.0)
    aim = c + unit(rng.normal(size=(N, 3))) * (r * rng.uniform(0, 1, N))[:, None]
    if name == "aimed":
        d = unit(aim - o)
    elif name == "grazing":
        side = unit(np.cross(d, rng.normal(size=(N, 3))))
        o = c + side * (r * (1 + rng.choice([-1, 1], N) * 10 ** rng.uniform(-9, -2, N)))[:, None] - d * rng.uniform(0.5, 3, N)[:, None]
    elif name == "surface":  # leaving, entering and tangential, from the surface
        o = c + unit(rng.normal(size=(N, 3))) * (r * (1 + rng.normal(size=N) * 1e-6))[:, None]
    elif name == "near_eps":  # a root at about 1e-4
        n = unit(rng.normal(size=(N, 3)))
        d = -unit(n + 0.5 * unit(rng.normal(size=(N, 3))))
        o = c + n * r[:, None] - d * (1e-4 * (1 + rng.normal(size=N) * 1e-4))[:, None]
    elif name == "lengths":
        d = unit(aim - o) * 10 ** rng.uniform(-2, 1, N)[:, None]
    elif name == "scales":
        k = 10 ** rng.uniform(-4, 5, N)
        d, o, c, r = unit(aim - o), o * k[:, None], c * k[:, None], r * k
    elif name == "degenerate":
        d = np.where(rng.random((N, 3)) < 0.4, 0.0, d)
        o = np.where(rng.random((N, 3)) < 0.3, c, o)
        r = np.where(rng.random(N) < 0.1, 0.0, r)
        d[:50], o[50:90], r[90:120] = np.nan, np.inf, np.inf
    return np.column_stack([o, d, c, r, tmin])


@pytest.mark.parametrize("name,undecided", [("free", 2e-4), ("aimed", 2e-3), ("grazing", 0.2), ("surface", 1.0),
                                            ("near_eps", 1.0), ("lengths", 1.0), ("scales", 1.0), ("degenerate", 1.0)])
def test_pairs_decide_as_fp64(name, undecided):
    rows = case(name)
    with np.errstate(all="ignore"):
        t, rem, code = roots(rows, 0)
        t64, rem64, code64 = roots(rows, 1)
    known = code != 2
    assert np.array_equal(code[known], code64[known])
    hit = known & (code == 1)
    assert np.array_equal(t[hit].view(np.uint32), t64[hit].view(np.uint32))
    assert np.array_equal(np.sign(rem[hit]), rem64[hit])
    assert (~known).mean() <= undecided, (~known).mean()
    assert hit.any()
    print(name, "undecided", (~known).mean(), "hits", hit.mean())
