"""Emitter lists as ckr_ltc_shade takes them apart: consecutive triangles that share the
edge from their first corner are shaded together, short lists sit in shared memory, and a
warp's triangles across the horizon are clipped lobe by lobe.  Lists of every kind against
the FP64 oracle.

The bar is absolute, in units of the emitters' summed radiance: a triangle's integral is a
sum of three or four edge integrals of at most pi, each within 6e-7 of its value in FP32
(theta / sin theta 4e-7, cross and dot products 2e-7), that may cancel to nearly nothing, so
its term of the pixel is within 4 pi 6e-7 / 2 pi = 1.2e-6 of its radiance; 2e-6 here.  Where an
edge passes so close to the point that FP32 does not resolve the angle, more: allowed for
1 % of the pixels, up to 1e-3.  A wrong corner, edge or colour moves most pixels by 1e-2."""
from __future__ import annotations

import numpy as np
import pytest

from chakumrender_gb300 import ckr
from test_ltc_host import oracle_ltc

pytestmark = pytest.mark.gpu


def check(got, ref, rgb):
    e = np.abs(got - ref).max(1) / rgb.sum(0).max()
    assert np.mean(e <= 2e-6) >= 0.99 and e.max() <= 1e-3, (np.mean(e <= 2e-6), e.max())


def shade(torch, g, tri, rgb):
    d = [torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda() for a in (g, tri, rgb)]
    out = torch.full((len(g), 3), -1.0, device="cuda")
    ckr.ltc_shade(d[0].data_ptr(), len(g), d[1].data_ptr(), d[2].data_ptr(), len(tri), out.data_ptr(),
                  torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def quads(n, seed):
    """Corners of n tilted quads, and a colour for each of their triangles."""
    rng = np.random.default_rng(seed)
    c = np.column_stack([rng.uniform(-2, 2, (n, 2)), rng.uniform(0.5, 3, n)])
    u, v = rng.normal(size=(n, 3)) * 0.4, rng.normal(size=(n, 3)) * 0.4
    p = np.stack([c - u - v, c + u - v, c + u + v, c - u + v], 1).astype(np.float32)
    return p, rng.uniform(1, 6, (2 * n, 3)).astype(np.float32)


def tris(p, order):
    return np.stack([p[:, o].reshape(len(p), 9) for o in order], 1).reshape(-1, 9)


FAN = ((0, 1, 2), (0, 2, 3))


@pytest.mark.parametrize("order", [FAN, ((0, 2, 3), (0, 1, 2)), ((0, 2, 1), (0, 3, 2)), ((0, 3, 2), (0, 2, 1)),
                                   ((1, 2, 0), (2, 3, 0)), ((0, 1, 2), (0, 1, 2)), ((0, 1, 2), (0, 3, 2))])
@pytest.mark.parametrize("n", [1, 5, 33])
def test_list_forms_vs_oracle(torch_cuda, order, n):
    g = ckr.gbuffer(7, 1500)
    p, rgb = quads(n, n)
    tri = tris(p, order)
    got = shade(torch_cuda, g, tri, rgb)
    check(got, oracle_ltc(g, tri, rgb), rgb)


@pytest.mark.parametrize("count", [1, 3, 63, 64, 65, 127])
def test_any_count_and_mixed_order(torch_cuda, count):
    """Odd counts end in a single triangle; a list offset by one pairs nothing (a quad's
    second triangle and the next one's first); 64 and 65 lie on both sides of shared memory."""
    g = ckr.gbuffer(9, 777)
    p, rgb = quads(64, 3)
    tri, rgb = tris(p, FAN), rgb
    for a, c in ((tri[:count], rgb[:count]), (tri[1:count + 1], rgb[1:count + 1])):
        got = shade(torch_cuda, g, a, c)
        check(got, oracle_ltc(g, a, c), c)
        # Rotated corners share no first corner with the next triangle.
        turned = np.concatenate([a[::2][:, [3, 4, 5, 6, 7, 8, 0, 1, 2]], a[1::2]])
        again = shade(torch_cuda, g, turned, np.concatenate([c[::2], c[1::2]]))
        check(again, oracle_ltc(g, turned, np.concatenate([c[::2], c[1::2]])), c)


@pytest.mark.parametrize("npx", [1, 31, 33, 64, 65, 2049])
def test_pixel_counts(torch_cuda, npx):
    g = ckr.gbuffer(5, 4096)
    p, rgb = quads(4, 8)
    tri = tris(p, FAN)
    full = shade(torch_cuda, g, tri, rgb)
    assert np.array_equal(shade(torch_cuda, g[:npx], tri, rgb), full[:npx])
