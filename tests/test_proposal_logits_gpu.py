"""Logits of any size: a softmax does not change when all its logits do by the same amount, and
nothing bounds the network's.  With all 64 outputs in use the kernels form exp(z) without the
maximum, which FP32 holds to |z| = 80; rows beyond take theirs from the maximum."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from chakumrender_gb300 import scene as S
from chakumrender_gb300.proposal import Proposal
from test_proposal import emulate, records, to_dev

pytestmark = pytest.mark.gpu
B4 = slice(O.MLP_NPARAMS - 64, O.MLP_NPARAMS)  # the output layer's biases


def probabilities(torch, params, rec, sd):
    prop = Proposal(S.RenderScene(sd), seed=7)
    prop.set_params(params.astype(np.float32))
    out = torch.zeros(len(rec), 64, dtype=torch.float16, device="cuda")
    prop.infer(to_dev(torch, rec).data_ptr(), len(rec), out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return out.double().cpu().numpy(), prop.encoding()


def room():
    return S.manylight_scene(S.manylight_spec(subdiv=2, width=96, height=54, nemit=256, nclusters=64))


@pytest.mark.parametrize("shift", [0, 64, 78, 80, 100, 300, 1e4, -60, -80, -100, -300, -1e4])
def test_inference(torch_cuda, shift):
    """Every row shifted; and every second output, so that both signs meet in one row."""
    sd, rng = room(), np.random.default_rng(3)
    rec = records(rng, 256, *(sd.tri9.reshape(-1, 3).min(0), sd.tri9.reshape(-1, 3).max(0)), 64)
    base = rng.normal(size=O.MLP_NPARAMS) * 0.15
    for which in (slice(0, 64), slice(0, 64, 2)):
        params = base.copy()
        params[B4][which] += shift
        got, (centre, scale, C) = probabilities(torch_cuda, params, rec, sd)
        # test_infer_vs_oracle's bar against the same emulation, which rounds the biases as the kernel.
        assert (0.5 * np.abs(got - emulate(params, rec, centre, scale, C)).sum(1)).max() < 1e-2


@pytest.mark.parametrize("shift", [81, -200])
def test_rows_beside_others(torch_cuda, shift):
    """A row's probabilities are its own, whatever the rest of its warp needs: W4 takes one
    hidden unit to all outputs, so that the rows' logits differ by more than the clamp allows."""
    sd, rng = room(), np.random.default_rng(3)
    rec = records(rng, 512, *(sd.tri9.reshape(-1, 3).min(0), sd.tri9.reshape(-1, 3).max(0)), 64)
    params = rng.normal(size=O.MLP_NPARAMS) * 0.15
    params[14464:18560].reshape(64, 64)[:, :8] += shift / 4
    prop = Proposal(S.RenderScene(sd), seed=7)
    prop.set_params(params.astype(np.float32))
    d = to_dev(torch_cuda, rec)
    all_, one = (torch_cuda.zeros(512, 64, dtype=torch_cuda.float16, device="cuda") for _ in range(2))
    prop.infer(d.data_ptr(), 512, all_.data_ptr())
    for i in range(512):
        prop.infer(d.data_ptr() + 48 * i, 1, one.data_ptr() + 128 * i)
    torch_cuda.cuda.synchronize()
    assert torch_cuda.equal(all_, one)


def test_rendering(torch_cuda):
    """Selection from two networks of equal softmaxes, one inside the clamp and one past it: the
    same frames but for the few light samples whose selection entry rounds the other way."""
    torch, sd = torch_cuda, room()
    scene, frames = S.RenderScene(sd), []
    for lo, hi in ((0.0, 12.0), (84.0, 96.0), (-112.0, -100.0)):
        params = np.zeros(O.MLP_NPARAMS, np.float32)
        params[B4] = lo
        params[B4][::5] = hi
        prop = Proposal(scene, seed=5, train=False)
        prop.set_params(params)
        rgb = torch.empty(54, 96, 3, device="cuda")
        prop.render(sd.camera, S.render_cfg(shader=S.SHADER_PATH_NEE, spp=2, max_depth=3, seed=4), rgb.data_ptr())
        torch.cuda.synchronize()
        frames.append(rgb.cpu().numpy())
    for f in frames[1:]:
        assert np.mean(np.all(np.abs(f - frames[0]) <= 1e-5 * np.abs(frames[0]) + 1e-7, axis=2)) > 0.9
