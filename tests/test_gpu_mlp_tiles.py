"""The cost model's forward and gradient at the edges of their tiles (128 and 64 samples) against float64."""
import os
import sys

import numpy as np
import pytest
import torch

from pumatch_b200 import learn

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))
import mlp_ref  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 128, 129, 1000, 9473, 60_001])
def test_forward_and_gradient(n):
    r = np.random.default_rng(n)
    w = (r.standard_normal(learn.NPARAM) * 0.2).astype(np.float32)
    x = (r.standard_normal((n, learn.NIN)) * 2 + 3).astype(np.float32)
    t = r.standard_normal((n, learn.NOUT)).astype(np.float32)
    m = learn.CostModel(0, seed=1)
    m.set_weights(w)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    y = m.forward_raw(xd).cpu().numpy()
    loss, grad = m.gradient(xd, td)
    want = mlp_ref.forward(w, x)
    wl, wg = mlp_ref.loss_and_grad(w, x, t)
    # 64-term dot products in float32 through three layers: under 200 roundings of 2^-24 on the way to an output
    tol = 200 * 2.0 ** -24
    assert np.linalg.norm(y - want) <= tol * np.linalg.norm(want)
    assert abs(loss - wl) <= 2 * tol * wl
    # (a unit within rounding of zero may switch for a sample: its share of the norm is of the same order)
    assert np.linalg.norm(grad - wg) <= 4 * tol * np.linalg.norm(wg)
    m.close()
