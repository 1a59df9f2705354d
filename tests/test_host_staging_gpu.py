"""The host-buffer queries' staging slots: rays in pageable memory are uploaded in chunks
that grow from an eighth of the full size, so calls of fewer rays than one full chunk use
several slots too.  Every result equals the device query's, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from chakumrender_gb300 import ckr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 131072, 131073, 400001, 917505, 1048577])
def test_pageable_rays_match_device(torch_cuda, n):
    torch = torch_cuda
    tri = ckr.icosphere(3)
    scene = ckr.Scene(tri)  # a fresh scene: its staging buffers are sized by this call
    rays = ckr.rays_incoherent([-1.5] * 3, [1.5] * 3, 3, n)
    ids, t = scene.trace_closest_host(rays)
    occ = scene.trace_any_host(rays)
    d_rays = torch.from_numpy(rays).cuda()
    d_id, d_t = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty(n, device="cuda")
    d_occ = torch.empty(n, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    scene.trace_closest(d_rays.data_ptr(), n, d_id.data_ptr(), d_t.data_ptr(), s)
    scene.trace_any(d_rays.data_ptr(), n, d_occ.data_ptr(), s)
    assert scene.check_device(s) == 0
    assert np.array_equal(ids.view(np.int32), d_id.cpu().numpy())
    assert np.array_equal(t, d_t.cpu().numpy()) and np.array_equal(occ, d_occ.cpu().numpy())
