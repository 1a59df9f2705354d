"""Emitters that ckr_ltc_shade passes over: a group (a triangle, or two that share an edge) whose
sphere lies below the horizons of all 32 pixels of a warp.  A pixel's value may not depend on
which pixels share its warp, so a frame whose surfaces face the emitters and face away from them by
whole warps equals, bit for bit, the same pixels shuffled, where nearly every warp has some
of each and takes every group.  (Bit for bit as long as a warp's queue of triangles across the
horizon holds them all, four triangles or few that cross: past that the order of a sum
depends on the warp.)  Over lists that end at and around the 32 triangles that a warp holds, in every
order of pairs, and for coordinates and colours at the ends of FP32; and against the FP64 oracle."""
from __future__ import annotations

import numpy as np
import pytest

from chakumrender_gb300 import ckr
from test_ltc_host import oracle_ltc
from test_ltc_pairs_gpu import FAN, check, quads, shade, tris

pytestmark = pytest.mark.gpu
ORDERS = [FAN, ((0, 2, 3), (0, 1, 2)), ((1, 2, 0), (2, 3, 0))]


def facing(n, seed):
    """G-buffer rows: runs of 64 pixels that share a normal within 15 degrees of +z or -z in
    turn, seen from 3 to 45 degrees of it (along the normal itself the reference divides by zero)."""
    rng = np.random.default_rng(seed)
    g = ckr.gbuffer(seed, n)
    runs = -(-n // 64)
    nn = np.column_stack([rng.uniform(-0.18, 0.18, (runs, 2)), np.where(np.arange(runs) % 2, -1.0, 1.0)])
    nn = np.repeat(nn / np.linalg.norm(nn, axis=1, keepdims=True), 64, 0)[:n]
    d = rng.normal(size=(n, 3))
    d -= nn * (d * nn).sum(1, keepdims=True)
    v = nn + rng.uniform(0.05, 1, (n, 1)) * d / np.linalg.norm(d, axis=1, keepdims=True)
    g[:, 0:3] = rng.uniform(-1, 1, (n, 3))
    g[:, 3] = rng.uniform(0.2, 1, n)
    g[:, 4:7], g[:, 8:11] = nn, v / np.linalg.norm(v, axis=1, keepdims=True)
    return g


def lights(n, seed, near):
    """Quads on both sides of the pixels; far off, where none crosses a horizon, or `near`."""
    p, rgb = quads(n, seed)
    if not near:
        p = p * np.float32(0.3) + np.array([0, 0, 9], np.float32)
    p[np.random.default_rng(seed).random(n) < 0.5] *= np.array([1, 1, -1], np.float32)
    return p, rgb


def same_shuffled(torch, g, tri, rgb):
    perm = np.random.default_rng(2).permutation(len(g))
    a, b = shade(torch, g, tri, rgb), shade(torch, g[perm], tri, rgb)
    assert np.array_equal(a[perm], b, equal_nan=True)
    return a


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("count", [1, 2, 30, 31, 32, 33, 34, 62, 63, 64, 65, 200])
def test_any_list(torch_cuda, order, count):
    p, rgb = lights(110, count, False)
    tri = tris(p, order)
    for a, c in ((tri[:count], rgb[:count]), (tri[1:count + 1], rgb[1:count + 1])):
        g = facing(1500, count)
        check(same_shuffled(torch_cuda, g, a, c), oracle_ltc(g, a, c), c)


@pytest.mark.parametrize("count", [3, 31, 32, 33, 64, 97])
def test_fans(torch_cuda, count):
    """Every triangle shares the edge with the next: pairs from the first on, also where the
    staged triangles end; and the list the other way round.  The upper half of the fans' pixels
    see it, the others do not."""
    w = np.linspace(0, 5, count + 1)
    rim = np.stack([np.cos(w), np.sin(w), 8 + 0.1 * np.sin(3 * w)], 1)
    tri = np.stack([np.concatenate([[0.1, 0.2, 7.9], rim[i], rim[i + 1]]) for i in range(count)]).astype(np.float32)
    rgb = np.random.default_rng(count).uniform(1, 6, (count, 3)).astype(np.float32)
    g = facing(1500, count)
    for a, c in ((tri, rgb), (tri[::-1].copy(), rgb[::-1].copy())):
        check(same_shuffled(torch_cuda, g, a, c), oracle_ltc(g, a, c), c)


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("seed", range(6))
def test_across_the_horizon(torch_cuda, order, seed):
    p, rgb = lights(2, seed, True)
    tri, g = tris(p, order), facing(3000, seed)
    check(same_shuffled(torch_cuda, g, tri, rgb), oracle_ltc(g, tri, rgb), rgb)


@pytest.mark.parametrize("scale", [1e-30, 1e-18, 1e-16, 1e16, 1e17, 3e18, 1e38])
@pytest.mark.parametrize("of", ["lights", "pixels", "both"])
def test_extreme_coordinates(torch_cuda, scale, of):
    p, rgb = lights(2, 1, True)
    p[:, :, 2] = np.abs(p[:, :, 2]) * np.array([[1], [-1]], np.float32)
    tri, g = tris(p, FAN), facing(1500, 3)
    if of != "pixels":
        tri = tri * np.float32(scale)
    if of != "lights":
        g[:, 0:3] *= np.float32(scale)
    same_shuffled(torch_cuda, g, tri, rgb)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 3e38])
@pytest.mark.parametrize("what", ["colour", "corner", "normal", "position"])
def test_no_numbers(torch_cuda, bad, what):
    p, rgb = lights(2, 1, True)
    p[:, :, 2] = np.abs(p[:, :, 2]) * np.array([[1], [-1]], np.float32)
    tri, g = tris(p, FAN), facing(1500, 3)
    if what == "colour":
        rgb[[0, 2]] = bad
    elif what == "corner":
        tri[[0, 2], 4] = bad
    else:
        g[::97, 4 if what == "normal" else 1] = bad
    same_shuffled(torch_cuda, g, tri, rgb)
