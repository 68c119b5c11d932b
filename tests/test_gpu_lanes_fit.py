"""Single- and multi-emitter fits by queue length: lane groups against one thread per ROI.

A call without a tuning table fits its queue with 32 or 16 lanes per ROI or
with one thread per ROI, by the queue's length (on the host, or on the device
where only the device knows it).  Every choice must give the one-thread rows
bit for bit (NaN as NaN), at and around the lengths where the choice changes,
down to one record, and on records whose fits clamp the background to zero.
"""
import numpy as np
import pytest

from qcstorm_b200 import lib as qlib
from qcstorm_b200 import synth
from test_gpu_flush_fit import edge_records

pytestmark = pytest.mark.gpu

# a wave of warps on 148 SMs (5 or, at 11x11, 4 blocks of 4 ROIs) and the longest queues of 16 lanes (the
# wave of 3 to 5 blocks of 8 ROIs times 8, 10 or 11 eighths)
WAVES = (2960, 4440, 4884, 5920, 7400, 8140)


def device(rec):
    import torch
    return torch.from_numpy(np.ascontiguousarray(rec).view(np.int16)).cuda()


@pytest.mark.parametrize("loc_type,R", [(0, 7), (1, 7), (0, 9), (1, 9), (0, 11), (1, 11), (0, 13)])
@pytest.mark.parametrize("n", [1, 3, 5] + [w + d for w in WAVES for d in (0, 1)])
def test_single_by_length(cuda_ok, loc_type, R, n):
    rec, para = edge_records(max(n, 2051), R, loc_type)
    check_single(rec, para, n)


# whole waves of one warp per scheduler (18,944 ROIs), and a rest beside them
@pytest.mark.parametrize("loc_type,R", [(0, 7), (1, 7), (0, 9), (1, 9), (0, 11), (1, 11), (0, 13)])
@pytest.mark.parametrize("n", [18944, 18945, 18946, 21312, 21313, 21904, 21906, 40000, 94721])
def test_single_rest(cuda_ok, loc_type, R, n):
    rec, para = edge_records(2051, R, loc_type)
    check_single(np.resize(rec, (n, rec.shape[1])), para, n)


def check_single(rec, para, n):
    import torch
    d = device(rec[:n])
    ctx = qlib.LocContext(para, n)
    rows = []
    for table in ([], [(1 << 30, 1)]):
        ctx.set_tuning(table)
        ctx.localize_device(d.data_ptr(), n)
        rows.append(ctx.read_rows()[0])
    # the count on the device, below its bound
    ctx.set_tuning([])
    count = torch.tensor([n - 1], dtype=torch.int32, device="cuda")
    wle = torch.from_numpy(ctx.wle(rec[:n])).cuda()
    torch.cuda.synchronize()
    ctx.localize_device_n(d.data_ptr(), wle.data_ptr(), count.data_ptr(), n)
    counted = ctx.read_rows()[0]
    ctx.close()
    np.testing.assert_array_equal(rows[0], rows[1])
    np.testing.assert_array_equal(counted, rows[1][:n - 1])


@pytest.mark.parametrize("loc_type,R", [(0, 7), (0, 11), (1, 7)])
@pytest.mark.parametrize("n", [1, 300, 12000])
def test_multi_by_length(cuda_ok, loc_type, R, n):
    rec, para, _ = synth.multi_rois(n, R=R, seed=80 + R)
    if loc_type == 1:
        para = para.copy(LocType=1, **synth.as3d_calibration())
    edge, _ = edge_records(max(n, 2051), R, 0)
    rec[::7, :R * R] = edge[:n][::7, :R * R]
    d = device(rec)
    out = []
    for limit in (0, -1):  # lane groups (two widths at 7x7), one thread per ROI
        ctx = qlib.LocContext(para, n)
        ctx.set_tuning_multi(limit, limit)
        ctx.localize_device(d.data_ptr(), n)
        out.append(ctx.read_rows())
        ctx.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
