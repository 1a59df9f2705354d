"""Frames from trees on both sides of the depth from which the renderer fetches rays dynamically
(kDynamicDepth, csrc/wavefront.cuh): the same triangles in leaves of one, two and three, whose trees
differ in depth, give the same hits and so the same frame (FP32 terms added in FP64 in any order,
rounded once: 2^-23), but for the few rays that meet an edge that two triangles share, where the
one tested first is kept."""
from __future__ import annotations

import numpy as np
import pytest

from chakumrender_gb300 import scene as S

pytestmark = pytest.mark.gpu


def box(extra):
    """The box scene with `extra` small triangles inside."""
    sd = S.load_xml(S.SCENES / "box.xml")
    rng = np.random.default_rng(extra)
    t = (rng.uniform(0.2, 0.8, (extra, 1, 3)) + rng.normal(size=(extra, 3, 3)) * 0.05).astype(np.float32)
    mats = [S.Material.from_buffer_copy(m) for m in sd.materials[:sd.nmat]]
    lights = [S.Light.from_buffer_copy(l) for l in sd.lights[:sd.nlights]]
    return S.SceneData(np.concatenate([sd.tri9, t.reshape(-1, 9)]), np.concatenate([sd.tri_mat, np.zeros(extra)]),
                       sd.sph4, sd.sph_mat, mats, lights, sd.camera)


@pytest.mark.parametrize("shader", [S.SHADER_PATH, S.SHADER_DIRECT_MIS])
def test_same_frame_at_any_depth(torch_cuda, shader):
    depths = set()
    for extra in (0, 6, 14, 26, 80):
        sd = box(extra)
        cam = sd.camera
        cam.width, cam.height = 97, 61
        frames = []
        for leaf in (0, 2, 1):
            scene = S.RenderScene(sd, leaf)
            depths.add(scene.info().max_depth)
            rgb = scene.render_host(cam, S.render_cfg(shader=shader, spp=3, max_depth=3, n_light=2, n_brdf=3, seed=5))
            assert scene.check_device() == 0
            frames.append(rgb.astype(np.float64))
        for f in frames[1:]:
            same = np.all(np.abs(f - frames[0]) <= 2.0**-23 * frames[0], axis=2)
            assert np.mean(same) > 0.995, np.mean(same)
    assert min(depths) < 4 <= max(depths), depths
