"""The training kernel at the edges of its 128-row tiles and of its grid: gradients against
the FP64 oracle for one row, around one tile, and for more tiles than blocks (accumulation
over a block's tiles), and a batch of no weight, which changes nothing."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from chakumrender_gb300 import scene as S
from chakumrender_gb300.proposal import Proposal
from test_proposal import records, to_dev

pytestmark = pytest.mark.gpu


def setup(seed):
    sd = S.manylight_scene(S.manylight_spec(subdiv=2, width=16, height=9, nemit=128, nclusters=64))
    prop = Proposal(S.RenderScene(sd), seed=7)
    rng = np.random.default_rng(seed)
    prop.set_params((rng.normal(size=O.MLP_NPARAMS) * 0.15).astype(np.float32))
    lo, hi = sd.tri9.reshape(-1, 3).min(0), sd.tri9.reshape(-1, 3).max(0)
    return prop, lambda n: records(rng, n, lo, hi, 64)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 152 * 128 - 1, 152 * 128 + 1, 2 * 152 * 128 + 130])
def test_gradients_at_tile_edges(torch_cuda, n):
    prop, make = setup(n)
    rec = make(n)
    rec[:, 7] = np.maximum(rec[:, 7], 0.05)
    loss, g = prop.gradients(to_dev(torch_cuda, rec).data_ptr(), n)
    centre, scale, _ = prop.encoding()
    loss_ref, g_ref = O.mlp_loss_grad(prop.params().astype(np.float64), rec, centre, scale, 64)
    # BF16 operands (2^-9 relative) against FP64: test_gradients_vs_oracle's bars.
    assert abs(loss - loss_ref) < 2e-2 * abs(loss_ref)
    x, y = g.astype(np.float64), g_ref
    assert x @ y / (np.linalg.norm(x) * np.linalg.norm(y)) > 0.99
    assert abs(np.linalg.norm(x) / np.linalg.norm(y) - 1) < 0.05


def test_a_batch_without_weight_changes_nothing(torch_cuda):
    prop, make = setup(3)
    rec = make(300)
    rec[:, 7] = 0
    before = prop.params()
    prop.train_step(to_dev(torch_cuda, rec).data_ptr(), len(rec))
    assert np.array_equal(prop.params(), before) and prop.status()[0] == 0
    rec = make(300)
    prop.train_step(to_dev(torch_cuda, rec).data_ptr(), len(rec))
    assert not np.array_equal(prop.params(), before)
