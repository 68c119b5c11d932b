"""Consecutive-frame merging and statistics with sort keys counted from the rows' ranges.

The keys hold only the digits that the rows' frames and positions span.  Rows
far outside the image, frames far from zero or far apart, groups of one row and
groups of one frame must give the oracle's links, merged rows, histograms and
neighbour counts, as rows of an ordinary movie do.
"""
import numpy as np
import pytest

import oracle_lib as O
from qcstorm_b200 import lib as qlib
from qcstorm_b200.abi import default_para
from qcstorm_b200.synth import blinking_rows

pytestmark = pytest.mark.gpu


def movie(case, loc_type):
    frames = 1 if case == "one_frame" else 9
    rows, counts = blinking_rows(n_emitters=300, frames=frames, seed=5, width=300, loc_type=loc_type,
                                 first_frame=3000000 if case == "late" else 1)
    if case in ("scattered", "outside"):
        rng = np.random.default_rng(6)
        k = rng.permutation(rows.shape[0])[:200]
        reach = 20000 if case == "scattered" else 9000
        rows[k, 1:3] = rng.uniform(-reach, reach, (200, 2))
    if case == "gap":
        rows[rows[:, 11] > 5, 11] += 65536
    if case == "one_row":
        rows, counts = rows[:1], np.array([1])
    sizes = np.add.reduceat(counts, np.arange(0, counts.size, 3)).astype(np.int32)
    return rows, sizes


CASES = ["plain", "late", "scattered", "outside", "gap", "one_row", "one_frame"]


# not "scattered": the oracle squares distances in 32-bit integers, as the
# reference does, and pairs rows whose squared distance overflows
@pytest.mark.parametrize("case", [c for c in CASES if c != "scattered"])
@pytest.mark.parametrize("loc_type,th_nm", [(0, 80.0), (1, 250.0)])
def test_merge(cuda_ok, case, loc_type, th_nm):
    rows, sizes = movie(case, loc_type)
    para = default_para(LocType=loc_type, ConsecFit_DistanceTh_nm=th_nm, PixelSize=100.0, QE=0.8)
    ora, ora_on = O.consec(para, rows, sizes, lib="oracle", gpu_rounding=1)
    cf = qlib.ConsecFit(capacity=int(max(sizes)))
    o = 0
    for g, n in enumerate(sizes):
        got, on = cf.fit(rows[o:o + n], para, is_end=g == len(sizes) - 1)
        o += n
        assert got.shape == ora[g].shape
        np.testing.assert_array_equal(got[:, 11], ora[g][:, 11])
        np.testing.assert_array_equal(got[:, 0] == 0, ora[g][:, 0] == 0)
        # the bounds of the ordinary movies: CRLB columns by another logf, the rest to float rounding
        np.testing.assert_allclose(got[:, 9:11], ora[g][:, 9:11], rtol=5e-3, equal_nan=True)
        keep = np.r_[0:9, 11]
        np.testing.assert_allclose(got[:, keep], ora[g][:, keep], rtol=2e-5, atol=1e-4, equal_nan=True)
        np.testing.assert_array_equal(on, ora_on[g])
    cf.close()


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("width,height", [(300, 300), (301, 47), (65535, 65535)])
def test_statistics(cuda_ok, case, width, height):
    rows, sizes = movie(case, 0)
    para = default_para(LocType=0, ImageWidth=width, ImageHigh=height)
    hist, means = O.stat(para, rows, sizes, lib="oracle")
    st = qlib.Statistics(capacity=int(max(sizes)))
    o = 0
    for g, n in enumerate(sizes):
        h, m = st.update(rows[o:o + n], para)
        o += n
        np.testing.assert_array_equal(h, hist[g])
        np.testing.assert_array_equal(m[6:7].view(np.uint32), means[g][6:7].view(np.uint32))  # density
        np.testing.assert_allclose(m, means[g], rtol=1e-5)
    st.close()
