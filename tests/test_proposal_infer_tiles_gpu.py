"""Inference on records (k_mlp_infer_rec, csrc/mlp.cu) at the edges of its rows, its 128-row
tiles, its seven tiles side by side in a block and its grid: a row's probabilities depend on
the row alone, so each equals, bit for bit, the one that a call of its tile alone gives (one
group of one block), and nothing is written past the last row; and fewer clusters than
outputs, against the arithmetic in numpy."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from chakumrender_gb300 import scene as S
from chakumrender_gb300.proposal import Proposal
from test_proposal import emulate, records, to_dev

pytestmark = pytest.mark.gpu
GUARD = 7.0  # no probability


def setup(nclusters, seed, scale=0.15):
    sd = S.manylight_scene(S.manylight_spec(subdiv=2, width=16, height=9, nemit=128, nclusters=nclusters))
    prop = Proposal(S.RenderScene(sd), seed=7)
    rng = np.random.default_rng(seed)
    params = (rng.normal(size=O.MLP_NPARAMS) * scale).astype(np.float32)
    prop.set_params(params)
    lo, hi = sd.tri9.reshape(-1, 3).min(0), sd.tri9.reshape(-1, 3).max(0)
    return prop, params, lambda n: records(rng, n, lo, hi, nclusters)


def infer(torch, prop, d_rec, n, calls_of=None):
    """Probabilities of n rows, in one call or in calls of `calls_of` rows, and four guard rows."""
    out = torch.full((n + 4, 64), GUARD, dtype=torch.float16, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    for at in range(0, n, calls_of or n):
        m = min(calls_of or n, n - at)
        prop.infer(d_rec.data_ptr() + 48 * at, m, out.data_ptr() + 128 * at, s)
    torch.cuda.synchronize()
    assert prop.status()[0] == 0
    return out


# Rows per SM and group: (tiles per SM, rows more or less).
@pytest.mark.parametrize("nclusters", [64, 33, 8])
@pytest.mark.parametrize("tiles,more", [(0, 1), (0, 31), (0, 33), (0, 127), (0, 128), (0, 129), (1, 1), (2, -1), (7, -1),
                                        (7, 1), (15, 33)])
def test_rows_do_not_depend_on_their_tile(torch_cuda, nclusters, tiles, more):
    torch = torch_cuda
    n = tiles * torch.cuda.get_device_properties(0).multi_processor_count * 128 + more
    prop, _, make = setup(nclusters, n)
    d_rec = to_dev(torch, make(n))
    got, ref = infer(torch, prop, d_rec, n), infer(torch, prop, d_rec, n, 128)
    assert torch.equal(got[:n], ref[:n])
    assert bool((got[n:] == GUARD).all()) and bool((ref[n:] == GUARD).all())


@pytest.mark.parametrize("nclusters", [1, 8, 32, 33, 63, 64])
def test_any_number_of_clusters(torch_cuda, nclusters):
    prop, params, make = setup(nclusters, nclusters)
    n = 300
    rec = make(n)
    got = infer(torch_cuda, prop, to_dev(torch_cuda, rec), n)[:n].double().cpu().numpy()
    centre, scale, C = prop.encoding()
    assert C == nclusters
    assert np.all(got[:, C:] == 0)
    # test_infer_vs_oracle's bar against the same emulation.
    assert (0.5 * np.abs(got - emulate(params, rec, centre, scale, C)).sum(1)).max() < 1e-2
