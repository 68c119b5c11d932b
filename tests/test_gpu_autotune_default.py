"""The autotuner against the choice by the queue's length that an untuned context makes.

A tuned context must not be slower than an untuned one, neither at a tuned size
nor between or above them, and a tuning file written for kernels that no longer
exist must not override the default.
"""
import numpy as np
import pytest

from qcstorm_b200 import lib as qlib
from qcstorm_b200 import synth
from test_gpu_lanes_fit import device

pytestmark = pytest.mark.gpu


def call_us(ctx, d, wle, n, counted=None):
    """Device time of one localization of n records (counted: the count on the device and its bound): the least
    of ten runs of ten."""
    import torch
    s = torch.cuda.Stream()
    best = float("inf")
    for _ in range(10):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record(s)
        for _ in range(10):
            if counted:
                ctx.localize_device_n(d.data_ptr(), wle.data_ptr(), counted[0].data_ptr(), counted[1], s.cuda_stream)
            else:
                ctx.localize_device(d.data_ptr(), n, wle.data_ptr(), s.cuda_stream)
        b.record(s)
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 100)
    return best


# above the tuned sizes, and between two of them: one thread per ROI takes 1.4 times as long, 16 lanes 1.16 times
@pytest.mark.parametrize("gen,R,tuned,n", [(synth.gs2d_rois, 11, 6000, 20000), (synth.gs2d_rois, 11, 65536, 20000),
                                           (synth.as3d_rois, 9, 30000, 1000)])
def test_tuned_context_is_no_slower(cuda_ok, gen, R, tuned, n):
    import torch
    rec, para, _ = gen(2000, R=R, seed=3)
    rec = np.resize(rec, (max(tuned, n), rec.shape[1]))
    d = device(rec)
    ctx = qlib.LocContext(para, rec.shape[0])
    wle = torch.from_numpy(ctx.wle(rec)).cuda()
    torch.cuda.synchronize()
    plain = call_us(ctx, d, wle, n)
    base = ctx.read_rows()[0]
    ctx.autotune(d.data_ptr(), wle.data_ptr(), tuned)
    got = call_us(ctx, d, wle, n)
    np.testing.assert_array_equal(ctx.read_rows()[0], base)
    ctx.close()
    assert got < 1.15 * plain


def test_tuning_files_of_both_versions(cuda_ok, tmp_path):
    _, para, _ = synth.multi_rois(10, R=11, seed=5)
    ctx, other = qlib.LocContext(para, 100), qlib.LocContext(para, 100)
    ctx.set_tuning([(1024, 8), (4096, 1)])
    ctx.set_tuning_multi(777, -1)
    now, old = tmp_path / "now.txt", tmp_path / "old.txt"
    ctx.save_tuning(now)
    other.load_tuning(now)
    assert other.tuning() == [(1024, 8), (4096, 1)] and other.tuning_multi() == (777, -1)
    text = now.read_text()
    assert text.startswith("qcstorm_b200_tuning 2\n")
    old.write_text(text.replace("qcstorm_b200_tuning 2", "qcstorm_b200_tuning 1", 1))
    other.load_tuning(old)  # read, its choices left
    assert other.tuning() == [] and other.tuning_multi() == (0, 0)
    old.write_text(text.replace("qcstorm_b200_tuning 2", "qcstorm_b200_tuning 3", 1))
    with pytest.raises(qlib.QcsError):
        other.load_tuning(old)
    wrong = qlib.LocContext(para.copy(ROISize=7), 100)
    old.write_text(text.replace("qcstorm_b200_tuning 2", "qcstorm_b200_tuning 1", 1))
    with pytest.raises(qlib.QcsError) as e:
        wrong.load_tuning(old)
    assert e.value.code == 6  # written for another shape, as before
    for c in (ctx, other, wrong):
        c.close()
