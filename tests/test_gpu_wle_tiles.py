"""WLE pre-pass on tiles of 64 records: ragged tiles, every ROI size, any record alignment.

The widths, neighbour distances and molecule types must equal the oracle's
(widths within 4e-7, the bound the pre-pass is held to on molecules' records)
whether the call ends inside a tile or not, and must not depend on whether the
records start on a 4-byte boundary; every fifth record is noise over the whole
range, whose widths are only held to the latter.
"""
import numpy as np
import pytest

from qcstorm_b200 import lib as qlib
from qcstorm_b200 import synth
import oracle_lib

pytestmark = pytest.mark.gpu


def estimate(ctx, para, ptr, n):
    import torch
    import ctypes as C
    out = torch.full((n, 6), float("nan"), device="cuda")
    torch.cuda.synchronize()
    qlib.check(qlib.load().qcs_wle_estimate_device(ctx.h, C.c_void_p(ptr), n, C.byref(para), C.c_void_p(out.data_ptr()),
                                                   None))
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("R", [5, 7, 9, 11, 13, 15, 17])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 193])
def test_ragged_tiles(cuda_ok, R, n):
    import torch
    rec, para, _ = synth.gs2d_rois(n, R=R, seed=90 + R)
    rng = np.random.default_rng(R)
    rec[::5, :R * R] = rng.integers(0, 65536, (rec[::5].shape[0], R * R))
    rec[:, R * R:R * R + 2] = rng.integers(10, 60, (n, 2))
    rec[:, R * R + 2] = 1 + np.arange(n) // 40
    order = rng.permutation(n)  # out of (frame, y, x) order
    rec, molecule = rec[order], order % 5 != 0
    buf = torch.zeros(rec.size + 1, dtype=torch.int16, device="cuda")
    ctx = qlib.LocContext(para, n)
    got = []
    for shift in (0, 1):
        buf[shift:shift + rec.size] = torch.from_numpy(rec.view(np.int16).reshape(-1)).cuda()
        got.append(estimate(ctx, para, buf.data_ptr() + 2 * shift, n))
    ctx.close()
    np.testing.assert_array_equal(got[0], got[1])
    ref = oracle_lib.wle(para, rec)
    np.testing.assert_array_equal(got[0][:, 0], ref[:, 0])
    np.testing.assert_allclose(got[0][molecule, 1:5], ref[molecule, 1:5], rtol=4e-7)
