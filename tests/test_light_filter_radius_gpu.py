"""A sphere light's radius counts by its square alone (Sphere::intersect, the light's
cone), so a negative one gives the frame of its magnitude: DIRECT_MIS may not leave out BRDF
samples that meet the sphere (may_meet_light, csrc/wavefront.cuh) near its rim.  Both frames
add the same FP32 terms in FP64, in an order that may differ, and round once: equal to
one unit in the last place, 2^-23."""
from __future__ import annotations

import numpy as np
import pytest

from chakumrender_gb300 import scene as S

pytestmark = pytest.mark.gpu


def frame(radius, spec):
    sd = S.load_xml(S.SCENES / "box.xml")
    mats = [S.Material.from_buffer_copy(m) for m in sd.materials[:sd.nmat]]
    for m in mats:
        if m.light_type == 0:
            m.spec, m.alpha = spec, 0.3
    em = S.Material.from_buffer_copy(sd.materials[int(sd.tri_mat[sd.lights[0].first])])
    em.radiance = S.F3(6.0, 9.0, 12.0)
    sph4 = np.concatenate([sd.sph4, [[0.3, 0.6, 0.4, radius]]])
    lights = [S.Light.from_buffer_copy(l) for l in sd.lights[:sd.nlights]]
    lights.append(S.Light(S.LIGHT_SPHERE, len(sd.sph4), 1, S.F3(0, 0, 0), S.F3(0, 0, 0), 0))
    sd = S.SceneData(sd.tri9, sd.tri_mat, sph4, np.concatenate([sd.sph_mat, [sd.nmat]]), mats + [em], lights, sd.camera)
    cam = sd.camera
    cam.width, cam.height = 77, 53
    scene = S.RenderScene(sd)
    rgb = scene.render_host(cam, S.render_cfg(shader=S.SHADER_DIRECT_MIS, spp=2, n_light=2, n_brdf=33, seed=5))
    assert scene.check_device() == 0 and np.all(np.isfinite(rgb))
    return rgb.astype(np.float64)


@pytest.mark.parametrize("spec", [0.0, 0.7])
def test_negative_radius_is_its_magnitude(torch_cuda, spec):
    a, b = frame(0.15, spec), frame(-0.15, spec)
    assert a.max() > 0.1
    assert np.all(np.abs(a - b) <= 2.0**-23 * a)
