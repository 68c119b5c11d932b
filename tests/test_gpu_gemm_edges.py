"""Training GEMMs at the edges of their tiles, chunks and splits.

A batch of n rows is the M of the forward and input-gradient products (tiles of
128 rows, the bias, ReLU and mask applied as they are stored) and the K of the
weight gradients (chunks of 128, split over blocks).  The bounds are those of
the same comparison at 512 rows: operands rounded to BF16 on both sides, sums
in another order.
"""
import os
import sys

import numpy as np
import pytest

from qcstorm_b200 import lib as qlib

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import qcs_net_oracle as NO  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 127, 129, 257, 1000, 2999])
@pytest.mark.parametrize("loc_type,R", [(0, 7), (1, 11)])
def test_gradient_matches_oracle(cuda_ok, loc_type, R, n):
    import torch
    rng = np.random.default_rng(n)
    nu = 6 if loc_type else 5
    width = NO.in_width(R)
    x = rng.normal(0, 0.5, (n, width)).astype(np.float32)
    t = rng.normal(0, 0.5, (n, nu)).astype(np.float32)
    v = (rng.random(n) < 0.9).astype(np.float32)
    v[0] = 1
    net = qlib.LearnedNet(batch=n, seed=3, loc_type=loc_type, roi_size=R)
    dx, dt, dv = (torch.from_numpy(a).cuda() for a in (x, t, v))
    y = net.forward(dx).cpu().numpy()
    loss = net.gradient(dx, dt, dv)
    g = net.grads()
    loss_o, g_o, y_o = NO.loss_and_grad(net.params(), x, t, v)
    assert np.max(np.abs(y - y_o)) <= 2e-3 * max(1.0, np.max(np.abs(y_o)))
    assert abs(loss - loss_o) <= 2e-3 * abs(loss_o)
    o = 0
    for size in (width * 128, 128, 128 * 128, 128, 128 * 8, 8):
        a, b = g[o:o + size], g_o[o:o + size]
        o += size
        assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b) + 1e-7, (size, np.linalg.norm(a - b))
    net.close()
