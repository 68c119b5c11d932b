"""Two- and three-emitter stages at the lengths where their kernel changes.

Up to one wave of warps (2,368 ROIs at four blocks an SM) a stage's queue takes a
warp per ROI, then half a warp at 7x7 and further rounds of warps at 11x11 up to
12,000 to 16,500 ROIs, then one thread per ROI, with lane groups again for some
lengths above its wave (18,944; 15,000 at 7x7 in a launch for many more).  Every record here is one that reaches the
stage, so that the queue's length is the call's; the fit ratios say so.  All must
give the one-thread rows, second emitters among them, bit for bit (NaN as NaN).
"""
import functools

import numpy as np
import pytest

from qcstorm_b200 import lib as qlib
from qcstorm_b200 import synth
from test_gpu_autotune_default import call_us
from test_gpu_lanes_fit import device

pytestmark = pytest.mark.gpu


def triplets(n, R, seed):
    """Records of three emitters about the centre, a third of a turn apart."""
    rng = np.random.default_rng(seed)
    sig, rad = rng.uniform(1.0, 1.4, n), rng.uniform(0.15 * R, 0.32 * R, n)
    at, turn = R / 2 + rng.uniform(-0.5, 0.5, (2, n)), rng.uniform(0, 2 * np.pi, n)
    mu = np.full((n, R, R), 30.0)
    for j in range(3):
        a = turn + j * 2 * np.pi / 3 + rng.uniform(-0.3, 0.3, n)
        mu += synth._gauss(R, at[0] + rad * np.cos(a), at[1] + rad * np.sin(a), sig, sig,
                           np.exp(rng.uniform(6, 9, n)) / (2 * np.pi * sig ** 2))
    return synth._records(np.minimum(rng.poisson(mu), 65535).astype(np.uint16), 1 + np.arange(n))


@functools.lru_cache(None)
def reaching(loc_type, R):
    """Records that reach the last stage (3E; AS3D: 2E), found one by one."""
    _, para, _ = synth.multi_rois(1, R=R)
    if loc_type == 1:
        para = para.copy(LocType=1, **synth.as3d_calibration())
    rec = triplets(1500, R, 5)
    ctx = qlib.LocContext(para, 1)
    stage = 1 if loc_type == 1 else 2
    keep = [i for i in range(rec.shape[0]) if ctx.localize(rec[i:i + 1])[1][stage] > 0]
    ctx.close()
    assert len(keep) >= 30
    return rec[keep], para


@pytest.mark.parametrize("loc_type,R", [(0, 7), (0, 11), (1, 7)])
@pytest.mark.parametrize("n", [2368, 2369, 4737, 12000, 12001, 13501, 16501, 18944, 18945, 20001, 25000, 30001])
def test_stage_lengths(cuda_ok, loc_type, R, n):
    base, para = reaching(loc_type, R)
    rec = np.resize(base, (n, base.shape[1]))
    rec[:, R * R + 2], rec[:, R * R + 3] = np.arange(n) & 0xFFFF, np.arange(n) >> 16  # a frame each: no neighbours
    d = device(rec)
    out = []
    # the default, lane groups whatever the length, one thread per ROI
    for limit in (0, 1 << 30, -1):
        ctx = qlib.LocContext(para, n)
        ctx.set_tuning_multi(limit, limit)
        ctx.localize_device(d.data_ptr(), n)
        rows, ratios = ctx.read_rows()
        assert ratios[1] == 1.0 and (loc_type == 1 or ratios[2] == 1.0)
        assert rows.shape[0] > n  # second emitters
        out.append(rows)
        ctx.close()
    np.testing.assert_array_equal(out[0], out[2])
    np.testing.assert_array_equal(out[1], out[2])


@pytest.mark.parametrize("loc_type,R", [(0, 7), (0, 11), (1, 7)])
@pytest.mark.parametrize("n,most", [(n, n) for n in (1000, 11000, 18000, 18950, 27000)] + [
    (n, 60000) for n in (14500, 16000, 20400, 27000)])
def test_default_is_no_slower_than_either_kernel(cuda_ok, loc_type, R, n, most):
    """The default against each kernel for the whole queue: wrong by at most a tenth of the call.  most: the
    call's bound, its count on the device where that is above n; the rows are those of one thread per ROI."""
    import torch
    base, para = reaching(loc_type, R)
    rec = np.resize(base, (n, base.shape[1]))
    rec[:, R * R + 2], rec[:, R * R + 3] = np.arange(n) & 0xFFFF, np.arange(n) >> 16
    d = device(rec)
    ctx = qlib.LocContext(para, most)
    wle = torch.from_numpy(ctx.wle(rec)).cuda()
    count = torch.tensor([n], dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    us, rows = [], []
    for limit in (0, 1 << 30, -1):
        ctx.set_tuning_multi(limit, limit)
        us.append(call_us(ctx, d, wle, n, None if most == n else (count, most)))
        rows.append(ctx.read_rows()[0])
    ctx.close()
    np.testing.assert_array_equal(rows[0], rows[2])
    np.testing.assert_array_equal(rows[1], rows[2])
    assert us[0] < 1.1 * min(us[1:])
