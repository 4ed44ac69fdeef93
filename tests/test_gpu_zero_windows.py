"""Raw Float32 imagery with areas of zeros on the general kernels (k_corr, k_corr_bf): windows of zeros have exactly zero
variance, whatever lies beside and above them, so their values are zero and not what an FP64 rounding makes
of them. Scene, points and bounds as for the one-tile kernel; surfaces of more than one tile, turned chips
among them, and surfaces too small for that kernel to pay.
"""

import numpy as np
import pytest

from test_gpu_fp_direct import compare, scene

pytestmark = pytest.mark.gpu

# (chip, radius x, radius y): more than one tile, then small.
CASES = [(32, 45, 45), (16, 48, 30), (24, 60, 12), (48, 40, 40), (8, 40, 70), (16, 4, 4), (12, 8, 8), (8, 10, 10)]


@pytest.mark.parametrize("chip,rx,ry", CASES)
@pytest.mark.parametrize("measure", ["zncc", "ncc"])
def test_direct(ar, O, gpu_lib, chip, rx, ry, measure):
    compare(ar, O, np.float32, chip, rx, ry, measure, None)


@pytest.mark.parametrize("chip,rx,ry", CASES)
def test_turned(ar, O, gpu_lib, chip, rx, ry):
    compare(ar, O, np.float32, chip, rx, ry, "zncc", (-4.0, 0.0, 3.0))


@pytest.mark.parametrize("chip,rx,ry", [(64, 32, 32), (64, 20, 12), (96, 16, 20), (128, 12, 12)])
@pytest.mark.parametrize("measure", ["zncc", "ncc"])
def test_split(ar, O, gpu_lib, chip, rx, ry, measure):
    """Large chips (split-BF16 products): the area of zeros lies beside the imagery and below it."""
    a, b, _ = scene(np.float32, chip + rx)
    a, b = np.pad(a, ((0, 250), (0, 250))), np.pad(b, ((0, 250), (0, 250)), mode="wrap")
    rng = np.random.default_rng(3)
    pts = ar.pointset(rng.uniform(60, 400, 200), rng.uniform(60, 400, 200), chip_size=chip,
                      search_radius_x=rx, search_radius_y=ry)
    p = ar.params(preprocess="none", quantize="none", similarity=measure, subpixel="none")
    got = ar.track(ar.ImagePair(a, b, np.ones(a.shape, bool), np.ones(a.shape, bool)), pts, p)
    want = O.track(a, b, {f: getattr(pts, f) for f in ar.points.FIELDS}, upsampling=1, measure=measure)
    m = ~np.isnan(want[0])
    assert m.sum() > 150 and np.array_equal(np.isnan(got.dx), ~m)
    assert np.abs(got.correlation[m] - want[2][m]).max() <= 1e-5
