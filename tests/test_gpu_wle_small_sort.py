"""WLE pre-pass of contexts on short batches in any order.

Up to 4,096 records out of (frame, y, x) order are sorted in one block, more by
the graph's sort.  Both sides of that line, powers of two and their neighbours,
records at equal positions, and batches in order between batches out of order
must give the rows of the ordered batch, whose neighbours are the oracle's.
"""
import numpy as np
import pytest

import oracle_lib as O
from qcstorm_b200 import lib as qlib
from test_gpu_wle_sort import crowded, orders

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 64, 1023, 1024, 1025, 2049, 4095, 4096, 4097])
@pytest.mark.parametrize("twins", [False, True])
def test_wle_short_batches(cuda_ok, n, twins):
    R = 7
    rec, para = crowded(max(n, 4), R, seed=n)
    rec = np.ascontiguousarray(rec[:n])
    if twins:
        rec[1::2, R * R:R * R + 4] = rec[:n // 2 * 2:2, R * R:R * R + 4]
    ctx = qlib.LocContext(para, capacity=5000)
    base = ctx.wle(rec)
    np.testing.assert_array_equal(base[:, 0], O.wle(para, rec)[:, 0])
    perms = orders(n, seed=1) if n > 3 else {"reversed": np.arange(n)[::-1].copy()}
    for name, perm in perms.items():
        got = ctx.wle(np.ascontiguousarray(rec[perm]))
        back = np.empty_like(got)
        back[perm] = got
        np.testing.assert_array_equal(back.view(np.uint32), base.view(np.uint32), err_msg=name)
        np.testing.assert_array_equal(ctx.wle(rec).view(np.uint32), base.view(np.uint32))
    ctx.close()
