"""Single-emitter calls by queue length captured in a CUDA graph.

A queue a little past whole waves of 18,944 ROIs has its rest fitted by a launch
beside the one-thread kernel (a programmatic launch, which a capture turns into a
programmatic edge).  Replays must give the one-thread rows bit for bit, and what
follows on the stream must find both kernels' rows: the captured step copies them.
"""
import numpy as np
import pytest

from qcstorm_b200 import lib as qlib
from test_gpu_flush_fit import edge_records
from test_gpu_lanes_fit import device

pytestmark = pytest.mark.gpu

MOST = 40000


class Rows:
    """A context's rows as torch sees foreign memory."""

    def __init__(self, ctx, n):
        self.__cuda_array_interface__ = {"shape": (n, 12), "typestr": "<f4", "data": (ctx.device_rows(), False), "version": 2}


@pytest.mark.parametrize("loc_type,R", [(0, 7), (1, 9), (0, 11)])
def test_rest_in_a_cuda_graph(cuda_ok, loc_type, R):
    import torch
    rec, para = edge_records(2051, R, loc_type)
    rec = np.resize(rec, (MOST, rec.shape[1]))
    d = device(rec)
    ctx = qlib.LocContext(para, MOST)
    wle = torch.from_numpy(ctx.wle(rec)).cuda()
    torch.cuda.synchronize()
    ctx.set_tuning([(1 << 30, 1)])
    ctx.localize_device(d.data_ptr(), MOST, wle.data_ptr())
    base = ctx.read_rows()[0]
    ctx.set_tuning([])
    s = torch.cuda.Stream()
    sh = s.cuda_stream
    rows, out = torch.as_tensor(Rows(ctx, MOST), device="cuda"), torch.zeros((MOST, 12), device="cuda")
    count = torch.zeros(1, dtype=torch.int32, device="cuda")

    def capture(step):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
            step()
            out.copy_(rows)
        return g

    def replay(g, n):
        with torch.cuda.stream(s):
            rows.zero_()
            for _ in range(2):
                g.replay()
        s.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy()[:n], base[:n])

    for n in (18945, 20000, MOST):  # the length known on the host
        ctx.localize_device(d.data_ptr(), n, wle.data_ptr(), sh)
        g = capture(lambda: ctx.localize_device(d.data_ptr(), n, wle.data_ptr(), sh))
        replay(g, n)
        del g
    g = capture(lambda: ctx.localize_device_n(d.data_ptr(), wle.data_ptr(), count.data_ptr(), MOST, sh))
    for n in (300, 7000, 18944, 18945, 20000, MOST):  # and on the device
        count.fill_(n)
        torch.cuda.synchronize()
        replay(g, n)
    del g
    ctx.close()
