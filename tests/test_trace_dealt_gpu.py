"""Small ray batches, which the launch deals out to the warps itself, against the same
rays inside a large batch, which fetches them dynamically: ids, t and occlusion bit for
bit, at the edges of the rule; and both kinds of launch inside a captured graph."""
from __future__ import annotations

import numpy as np
import pytest

from chakumrender_gb300 import ckr

pytestmark = pytest.mark.gpu
BIG = 400000  # more rays than resident lanes on any part with up to 390 SMs


def query(torch, scene, d_rays, n, out, stream):
    scene.trace_closest(d_rays.data_ptr(), n, out[0].data_ptr(), out[1].data_ptr(), stream)
    scene.trace_any(d_rays.data_ptr(), n, out[2].data_ptr(), stream)


def buffers(torch, n):
    return (torch.full((n,), -7, dtype=torch.int32, device="cuda"), torch.zeros(n, device="cuda"),
            torch.full((n,), 9, dtype=torch.uint8, device="cuda"))


def setup(torch, spheres):
    sph = np.array([[0.2, 0.1, 1.3, 0.4], [-1.2, 0.3, 0.0, 0.5]], np.float32) if spheres else None
    scene = ckr.Scene(ckr.icosphere(4), sph)
    rays = np.concatenate([ckr.rays_incoherent([-1.6] * 3, [1.6] * 3, 5, BIG // 2, 0.1, 3.0),
                           ckr.rays_pinhole([0, 0, 3], [0, 0, 0], [0, 1, 0], 40.0, 500, 400)])
    return scene, torch.from_numpy(rays[np.random.default_rng(1).permutation(BIG)]).cuda()


@pytest.mark.parametrize("spheres", [False, True])
def test_few_rays_match_many(torch_cuda, spheres):
    torch = torch_cuda
    scene, d_rays = setup(torch, spheres)
    s = torch.cuda.current_stream().cuda_stream
    ref = buffers(torch, BIG)
    query(torch, scene, d_rays, BIG, ref, s)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    lanes = sms * 8 * 4 * 32  # eight resident blocks of four warps
    for n in (1, 3, 31, 33, 127, 129, sms * 8, sms * 8 + 1, 5000, lanes // 2 + 7, lanes - 1, lanes, lanes + 1):
        out = buffers(torch, n + 5)
        query(torch, scene, d_rays, n, out, s)
        for a, b, untouched in zip(out, ref, (-7, 0, 9)):
            assert torch.equal(a[:n], b[:n]), n
            assert bool((a[n:] == untouched).all()), n
    assert scene.check_device(s) == 0


@pytest.mark.parametrize("n", [100, 300000])
def test_inside_a_captured_graph(torch_cuda, n):
    torch = torch_cuda
    scene, d_rays = setup(torch, True)
    ref, out = buffers(torch, n), buffers(torch, n)
    query(torch, scene, d_rays, n, ref, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        query(torch, scene, d_rays, n, out, torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        out[0].fill_(-7)
        g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(out, ref))
