"""Which kernel a UInt8 pass runs on: k_corr_tc2 where its plan fits (surfaces up to 64 x 64, the chip operand
whole), else k_corr_tc (larger chips and surfaces), else the CUDA-core kernel, as the context's table of large
passes lists it; nothing is listed with the table off."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(16, 8, 8, "k_corr_tc2"), (32, 25, 25, "k_corr_tc2"), (32, 32, 32, "k_corr_tc2"),
         (64, 32, 32, "k_corr_tc2"), (32, 33, 10, "k_corr_tc"), (32, 10, 33, "k_corr_tc"), (16, 44, 44, "k_corr_tc"),
         (128, 6, 6, "k_corr_tc"), (128, 25, 25, "k_corr_tc"), (64, 48, 48, "k_corr_tc")]


@pytest.mark.parametrize("chip,rx,ry,kernel", CASES)
def test_first_plan_that_fits(ar, gpu_lib, chip, rx, ry, kernel):
    rng = np.random.default_rng(0)
    a = rng.integers(0, 256, (420, 420)).astype(np.uint8)
    n = 8192
    pts = ar.pointset(rng.uniform(0, 420, n), rng.uniform(0, 420, n), chip_size=chip, search_radius_x=rx,
                      search_radius_y=ry)
    p = ar.params(preprocess="none", quantize="none", subpixel="none")
    L = ar._lib
    for keep in (1, 0):
        ctx = L.Context(0)
        try:
            ctx.set_option(L.AR_OPT_AUTOTUNE, keep)
            ar.track(ar.ImagePair(a, a), pts, p, ctx=ctx)
            want = [{"chip": [chip, chip], "surface": [2 * ry, 2 * rx], "kernel": kernel}] if keep else []
            assert ctx.tuned() == want
        finally:
            ctx.close()
