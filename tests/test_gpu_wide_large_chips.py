"""k_corr_tc on large chips with surfaces beyond 64 x 64, whose box sums are computed in stripes
of surface rows: bit-identical to the CUDA-core kernel (exact integer numerators and sums, the
same FP64 normalisation)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (chip, rx, ry): surfaces just past 64 columns or rows, the radii of the batching configuration,
# remainders of the 16-row stripes, the four-row slide and the 128-column prefix passes, chip
# areas that are not powers of two.
CASES = [(64, 48, 48), (64, 33, 50), (64, 64, 34), (96, 40, 36), (100, 37, 35), (128, 48, 48),
         (128, 33, 33), (128, 34, 47), (128, 20, 41), (200, 33, 10)]


@pytest.mark.parametrize("chip,rx,ry", CASES)
@pytest.mark.parametrize("measure", ["zncc", "ncc"])
def test_striped_box_sums_identical(ar, gpu_lib, chip, rx, ry, measure):
    ref, sec = ar.synthetic.shifted_pair(520, (-5.3, 3.7), seed=chip + rx, dtype=np.uint8)
    sv = np.ones(ref.shape, bool)
    sv[200:260, 100:300] = False
    rng = np.random.default_rng(chip * 7 + ry)
    # Scattered points (some windows leave the image), then columns of points a few rows apart,
    # whose sums carry over from one to the next.
    x = np.concatenate([rng.uniform(0, 520, 60), np.repeat(rng.uniform(200, 320, 6), 12)])
    y = np.concatenate([rng.uniform(0, 520, 60),
                        np.concatenate([180 + np.cumsum(rng.integers(1, 24, 12)) for _ in range(6)])])
    pts = ar.pointset(x, y, chip_size=chip, search_radius_x=rx, search_radius_y=ry,
                      dx_prior=np.round(rng.uniform(-3, 3, x.size)), dy_prior=0.0)
    pair = ar.ImagePair(ref, sec, None, sv)
    p = ar.params(preprocess="none", quantize="none", similarity=measure, upsampling=16)
    ctx = ar._lib.default_context()
    got = {}
    try:
        for kernel in (1, 0):
            ctx.set_option(ar._lib.AR_OPT_UINT8_KERNEL, kernel)
            got[kernel] = ar.track(pair, pts, p, ctx=ctx)
    finally:
        ctx.set_option(ar._lib.AR_OPT_UINT8_KERNEL, -1)
    for name in ("dx", "dy", "correlation"):
        a, b = (getattr(got[k], name).view(np.uint32) for k in (1, 0))
        assert np.array_equal(a, b), name
    assert np.array_equal(got[1].searched, got[0].searched)
    assert np.count_nonzero(~np.isnan(got[1].dx)) > x.size // 2
