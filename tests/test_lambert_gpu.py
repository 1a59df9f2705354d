"""Vertices without a specular part (is_lambert, csrc/shading_device.cuh): their BRDF and pdf
are taken as 1 / pi and cos / pi, and the analytic shaders leave out their residual, an exact
zero.  A specular coefficient of 2e-38 keeps every vertex on the general evaluation and adds
nothing that FP32 can hold, so both frames are the same sums on the same random streams: at
the edges of the rule's roughness and refraction, and past them.

The bar: a pixel is at most 64 terms of one sign added in an order that may differ between
two launches, so two such sums are within 2 * 64 * 2^-24 = 7.7e-6 of each other; the residuals
the general evaluation keeps are below 1e-20."""
from __future__ import annotations

import numpy as np
import pytest

from chakumrender_gb300 import scene as S

pytestmark = pytest.mark.gpu


def frame(spec, shader, alpha, ior):
    sd = S.load_xml(S.SCENES / "box.xml")
    for m in sd.materials[:sd.nmat]:
        if m.light_type == 0:
            m.spec, m.alpha = spec, alpha
            m.int_ior, m.ext_ior = ior
    cam = sd.camera
    cam.width, cam.height = 77, 53
    scene = S.RenderScene(sd)
    rgb = scene.render_host(cam, S.render_cfg(shader=shader, spp=3, n_light=2, n_brdf=5, seed=5)).astype(np.float64)
    assert scene.check_device() == 0 and np.all(np.isfinite(rgb))
    return rgb


@pytest.mark.parametrize("shader", [S.SHADER_PATH, S.SHADER_DIRECT_MIS, S.SHADER_DIRECT_MISCV, S.SHADER_EXPLICIT])
@pytest.mark.parametrize("alpha,ior", [(1.0, (1e4, 1.0)), (0.01, (1.5, 1.0)), (0.0099, (1.5, 1.0)), (1000.0, (1.0, 1.0)),
                                       (0.3, (1e5, 1e-3))])
def test_same_frame_as_the_general_evaluation(torch_cuda, shader, alpha, ior):
    a, b = frame(0.0, shader, alpha, ior), frame(2e-38, shader, alpha, ior)
    assert b.max() > 0.1
    assert np.all(np.abs(a - b) <= 7.7e-6 * np.abs(b) + 1e-20)
