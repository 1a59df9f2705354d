"""The training kernel's rows, one by one at the edges of its 128-row tiles and of its grid: one
record holds all of a batch's weight but 1e-8 of it, so the batch's gradient is that record's alone,
and a row that is missing, counted twice or lost with its tile changes it by its whole size; rows
past the last do not take part; and steps inside a captured graph, whose kernels overlap by
programmatic launches there too."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from chakumrender_gb300 import scene as S
from chakumrender_gb300.proposal import Proposal
from test_proposal import records, to_dev

pytestmark = pytest.mark.gpu


def setup(seed):
    sd = S.manylight_scene(S.manylight_spec(subdiv=2, width=64, height=36, nemit=128, nclusters=64))
    scene = S.RenderScene(sd)
    prop = Proposal(scene, seed=7)
    rng = np.random.default_rng(seed)
    params = (rng.normal(size=O.MLP_NPARAMS) * 0.15).astype(np.float32)
    prop.set_params(params)
    lo, hi = sd.tri9.reshape(-1, 3).min(0), sd.tri9.reshape(-1, 3).max(0)
    return sd, prop, params, lambda n: records(rng, n, lo, hi, 64)


# Rows: a full grid's tiles and some more or less.  The heavy row: the first, the last, the
# first tile's last, the first of block 0's second tile.
SIZES = [(0, 1), (0, 127), (0, 128), (0, 129), (0, 257), (1, -1), (1, 1), (2, 130)]


@pytest.mark.parametrize("tiles,more,heavy", [(t, m, h) for h in (0, -1, 127, "second") for t, m in SIZES
                                              if not (h == 127 and t == 0 and m < 128 or h == "second" and (t, m) < (1, 1))])
def test_every_row_counts_once(torch_cuda, tiles, more, heavy):
    torch = torch_cuda
    full = torch.cuda.get_device_properties(0).multi_processor_count * 128
    n = tiles * full + more
    row = n - 1 if heavy == -1 else full if heavy == "second" else heavy
    _, prop, params, make = setup(n)
    rec = make(n + 300)
    rec[:, 7] = np.clip(rec[:, 7], 0.05, 10)
    rec[row, 7] = 1e9 * n  # the weights' FP32 sum is this one
    rec[n:, 7] = 1e10 * n  # not this batch's
    d = to_dev(torch, rec)
    loss, g = prop.gradients(d.data_ptr(), n)
    loss1, alone = prop.gradients(d.data_ptr() + 48 * row, 1)
    # The others' share is at most 1e-8 of the weight, a few times that of the gradient; the
    # sums over 128 rows a tile and three tiles round by 2^-24 each, a few 1e-7 in all.
    assert np.abs(alone).max() > 1e-3 and np.abs(g - alone).max() <= 2e-6 * np.abs(alone).max()
    assert abs(loss - loss1) <= 1e-5 * abs(loss1)
    d[n:] = 0
    assert np.array_equal(prop.gradients(d.data_ptr(), n)[1], g)


@pytest.mark.parametrize("n", [1, 4096, 30000])
def test_steps_inside_a_captured_graph(torch_cuda, n):
    """Three steps and an inference behind them, captured and replayed, equal the same calls
    made one after the other, bit for bit."""
    torch = torch_cuda
    _, prop, params, make = setup(5)
    rec = make(3 * n)
    rec[:, 7] = np.maximum(rec[:, 7], 0.05)  # no batch without weight
    d = to_dev(torch, rec)
    probs = [torch.zeros(n, 64, dtype=torch.float16, device="cuda") for _ in range(2)]

    def steps(out):
        s = torch.cuda.current_stream().cuda_stream
        for k in range(3):
            prop.train_step(d.data_ptr() + 48 * n * k, n, s)
        prop.infer(d.data_ptr(), n, out.data_ptr(), s)

    steps(probs[0])
    torch.cuda.synchronize()
    eager = prop.params()
    prop.set_params(params)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        steps(probs[1])
    assert np.array_equal(prop.params(), params)  # captured, not run
    g.replay()
    torch.cuda.synchronize()
    assert prop.status()[0] == 0 and not np.array_equal(eager, params)
    assert np.array_equal(prop.params(), eager) and torch.equal(*probs)


@pytest.mark.parametrize("train", [False, True])
def test_learned_frame_inside_a_captured_graph(torch_cuda, train):
    """A frozen frame captured and replayed adds the same terms as the frame by itself (in FP64, in
    any order, rounded once: 2^-23); one that trains leaves a trained network and a finite frame."""
    torch = torch_cuda
    sd, prop, params, _ = setup(6)
    prop.set_training(train)
    cfg = S.render_cfg(shader=S.SHADER_PATH_NEE, spp=2, max_depth=3, seed=4)
    frames = [torch.zeros(36, 64, 3, device="cuda") for _ in range(2)]
    prop.render(sd.camera, cfg, frames[0].data_ptr(), None, torch.cuda.current_stream().cuda_stream)  # workspaces
    torch.cuda.synchronize()
    prop.set_params(params)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        prop.render(sd.camera, cfg, frames[1].data_ptr(), None, torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        frames[1].zero_()
        g.replay()
        torch.cuda.synchronize()
        a, b = (f.double().cpu().numpy() for f in frames)
        assert prop.status()[0] == 0 and np.all(np.isfinite(b)) and b.max() > 0
        if not train:
            assert np.all(np.abs(a - b) <= 2.0**-23 * a)
    assert np.array_equal(prop.params(), params) != train
