"""The BRDF samples that the direct-light shaders cut down to those whose direction may
meet a light (may_meet_light, csrc/wavefront.cuh), 32 at a time: the frame equals the
FP64 oracle's, which evaluates every sample on the same random streams, for sample counts
at the edges of the groups and for lights whose bounding sphere holds the shaded points."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from chakumrender_gb300 import scene as S
from scene_io import rel_mse

pytestmark = pytest.mark.gpu
BAR = 1e-4  # of test_render_gpu.py's direct-light cases: FP32 against FP64, same streams


def box(extra: bool):
    """The box scene; `extra`: with a second mesh light, two small triangles on opposite
    walls, so that its bounding sphere holds most of the box."""
    sd = S.load_xml(S.SCENES / "box.xml")
    if not extra:
        return sd
    n = len(sd.tri9)
    tri = np.array([[0.002, 0.2, 0.3, 0.002, 0.3, 0.3, 0.002, 0.25, 0.4],
                    [0.998, 0.7, 0.5, 0.998, 0.8, 0.6, 0.998, 0.8, 0.4]], np.float32)
    mats = [S.Material.from_buffer_copy(m) for m in sd.materials[:sd.nmat]]
    em = S.Material.from_buffer_copy(sd.materials[int(sd.tri_mat[sd.lights[0].first])])
    em.radiance = S.F3(6.0, 9.0, 12.0)
    lights = [S.Light.from_buffer_copy(l) for l in sd.lights[:sd.nlights]]
    lights.append(S.Light(S.LIGHT_MESH, n, 2, S.F3(0, 0, 0), S.F3(0, 0, 0), 0))
    return S.SceneData(np.concatenate([sd.tri9, tri]), np.concatenate([sd.tri_mat, [sd.nmat, sd.nmat]]), sd.sph4,
                       sd.sph_mat, mats + [em], lights, sd.camera)


@pytest.mark.parametrize("shader", [S.SHADER_DIRECT_MISCV, S.SHADER_DIRECT_MIS])
@pytest.mark.parametrize("n_light,n_brdf,extra", [(1, 1, False), (2, 31, True), (1, 32, False), (3, 33, True),
                                                  (33, 65, False)])
def test_filtered_samples_vs_oracle(torch_cuda, shader, n_light, n_brdf, extra):
    sd = box(extra)
    cam = sd.camera
    cam.width, cam.height = 61, 45
    cfg = S.render_cfg(shader=shader, spp=2, n_light=n_light, n_brdf=n_brdf, seed=7)
    scene = S.RenderScene(sd)
    g = scene.render_host(cam, cfg).astype(np.float64)
    assert scene.check_device() == 0 and np.all(np.isfinite(g))
    o = O.render(sd, cam, cfg)
    e = rel_mse(g, o)
    assert e <= BAR, e
    assert abs(g.mean() - o.mean()) <= 1e-3 * o.mean()
