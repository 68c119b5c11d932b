"""The one-thread single-emitter fit where its flushing exp and log could show.

fit_single_kernel takes exp and log without subnormal handling where the
background or the exponents' range allows it, and the general forms for a warp
where some ROI does not.  Records whose fits clamp the background to zero, push
widths and positions far out, or hold constant, zero or saturated pixels reach
both sides of that line.  fit_lanes_kernel, which evaluates the same
terms with other code, must give the same rows bit for bit (NaN as NaN), on
records at 4-byte and at 2-byte boundaries.
"""
import numpy as np
import pytest

from qcstorm_b200 import lib as qlib
from qcstorm_b200 import synth
from test_gpu_group_fit import CASES, random_wle

pytestmark = pytest.mark.gpu


def edge_records(n, R, loc_type):
    rec, para, _ = synth.gs2d_rois(n, R=R, seed=60 + R) if loc_type == 0 else synth.as3d_rois(n, R=R, seed=70 + R)
    rng = np.random.default_rng(R)
    P, off = R * R, int(para.Offset)
    c = np.arange(R) - R // 2
    psf = np.exp(-(c[:, None] ** 2 + c[None, :] ** 2) / 2 / 1.2 ** 2).reshape(-1)
    k = n // 8
    rec[:k, :P] = off + rng.integers(0, 3, (k, P))
    rec[k:2 * k, :P] = off
    rec[k:2 * k, P // 2] = 30000
    rec[2 * k:3 * k, :P] = off + rng.poisson(np.exp(rng.uniform(1, 9, (k, 1))) * psf)  # no background
    rec[3 * k:4 * k, :P] = rng.integers(0, 65536, (k, P))
    rec[4 * k:4 * k + 40, :P] = 65535
    rec[4 * k + 40:4 * k + 80, :P] = 0
    return rec, para


@pytest.mark.parametrize("loc_type,R", CASES)
@pytest.mark.parametrize("n,shift", [(2051, 0), (2051, 1), (33, 0), (1, 0)])
def test_flushing_fit_equals_general_fit(cuda_ok, loc_type, R, n, shift):
    import torch
    rec, para = edge_records(max(n, 2051), R, loc_type)
    rec = rec[:: max(1, rec.shape[0] // n)][:n]
    buf = torch.zeros(rec.size + 2, dtype=torch.int16, device="cuda")
    buf[shift:shift + rec.size] = torch.from_numpy(np.ascontiguousarray(rec).view(np.int16).reshape(-1)).cuda()
    wle = torch.from_numpy(random_wle(n, R, seed=R)).cuda()
    rows = []
    for fit in (qlib.fit_single_device, qlib.fit_single_group_device):
        out = torch.full((n, 12), float("nan"), device="cuda")
        fit(loc_type, para, buf.data_ptr() + 2 * shift, wle.data_ptr(), n, out.data_ptr())
        torch.cuda.synchronize()
        rows.append(out.cpu().numpy())
    np.testing.assert_array_equal(rows[0], rows[1])
