"""Raw Float32 imagery with areas of zeros on the general kernel (k_corr): windows of zeros have exactly zero
variance, whatever lies beside and above them, so their values are zero and not what an FP64 rounding makes
of them. Scene, points and bounds as for the one-tile kernel; surfaces of more than one tile, turned chips
among them, and surfaces too small for that kernel to pay.
"""

import numpy as np
import pytest

from test_gpu_fp_direct import compare

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
