"""How the shading kernels split their rows: a large LTC frame (two tiles of 64 pixels to a
block) equals, bit for bit, the same pixels shaded in calls that the resident blocks hold; and
frames around the first rows of all shading warps (the rest come from a counter) equal the FP64
oracle's on the same random streams."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from chakumrender_gb300 import ckr, scene as S
from scene_io import rel_mse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [-1, 0, 1, 63, 65])
def test_ltc_large_frame_equals_its_parts(torch_cuda, extra):
    torch = torch_cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n, part = 2 * 8 * sms * 64 + extra, 64 * 1024
    g = torch.Generator(device="cuda").manual_seed(3)
    buf = torch.rand(n, 12, device="cuda", generator=g) * 2 - 1
    for c in (4, 8):  # normal, view direction
        v = torch.nn.functional.normalize(buf[:, c:c + 3], dim=1)
        buf[:, c:c + 3] = v
    buf[:, 8:11] *= torch.sign((buf[:, 4:7] * buf[:, 8:11]).sum(1, keepdim=True))
    buf[:, 3] = buf[:, 3].abs().clamp_min(0.05)
    buf[:, 7], buf[:, 11] = buf[:, 7].abs(), buf[:, 11].abs()
    tri = (torch.rand(6, 9, device="cuda", generator=g) * 4 - 2).contiguous()
    col = torch.rand(6, 3, device="cuda", generator=g)
    whole, parts = torch.empty(n, 3, device="cuda"), torch.empty(n, 3, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    ckr.ltc_shade(buf.data_ptr(), n, tri.data_ptr(), col.data_ptr(), 6, whole.data_ptr(), stream)
    for a in range(0, n, part):
        ckr.ltc_shade(buf[a:].data_ptr(), min(part, n - a), tri.data_ptr(), col.data_ptr(), 6, parts[a:].data_ptr(), stream)
    torch.cuda.synchronize()
    assert torch.equal(whole.view(torch.int32), parts.view(torch.int32))


@pytest.mark.parametrize("width,height", [(456, 256), (457, 257)])
def test_rows_from_the_counter(torch_cuda, width, height):
    # 152 SMs x 6 blocks x 128 rows are 456 x 256.
    sd = S.load_xml(S.SCENES / "box.xml")
    cam = sd.camera
    cam.width, cam.height = width, height
    cfg = S.render_cfg(shader=S.SHADER_DIRECT_MISCV, spp=1, n_light=1, n_brdf=2, seed=9)
    scene = S.RenderScene(sd)
    g = scene.render_host(cam, cfg).astype(np.float64)
    assert scene.check_device() == 0 and np.all(np.isfinite(g))
    assert rel_mse(g, O.render(sd, cam, cfg)) <= 1e-4  # the direct-light bar of FP32 against FP64
