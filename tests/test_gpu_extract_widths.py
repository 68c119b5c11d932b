"""Extraction over image widths on both sides of the eight-pixel detection rule.

GS2D with multi-emitter fitting tests eight pixels a thread where the width is
a multiple of 8, and tiles otherwise; the background sums four-byte pairs and
divides by three without a division.  Widths below, at and past a block's 256
columns, heights that leave part of a block, batches of ragged frames, and
pixels up to 65,535 (the largest border sums) must all give the oracle's
records bit for bit, in its order.
"""
import numpy as np
import pytest

import oracle_lib as O
from qcstorm_b200 import synth
from test_gpu_extract import DEVICE_MODE, check_wle, run_product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [64, 104, 250, 256, 264, 513, 520])
@pytest.mark.parametrize("height,frames,batch,R,gain", [(41, 3, 2, 5, 1), (64, 2, 2, 7, 1), (97, 2, 1, 9, 60)])
def test_records_match_oracle(cuda_ok, width, height, frames, batch, R, gain):
    fr, para, _ = synth.frames(frames, width=width, height=height, density=max(20, width * height // 500), seed=width + height)
    fr = np.minimum(fr.astype(np.int64) * gain, 65535).astype(np.uint16)
    assert gain == 1 or (fr == 65535).any()
    para.LocType, para.MultiEmitterFitEn, para.ROISize = 0, 1, R
    rois, wle, span, dropped = run_product(fr, para, batch, start_frame=7)
    ro, wo, g0, g1 = O.extract(para, fr, batch, start_frame=7, flags=DEVICE_MODE)
    assert dropped == 0 and ro.shape[0] > 0
    assert np.array_equal(rois, ro)
    assert span == (g0, g1)
    assert np.array_equal(wle[:, 0], wo[:, 0])  # nearest neighbours
    if gain == 1:
        check_wle(para, rois, wle, wo)
