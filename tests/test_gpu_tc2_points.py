"""k_corr_tc2 against the CUDA-core kernel, bit for bit, where its shortcuts can go wrong: windows
without variance (estimates left to the exact evaluation) and all-zero ones, several equal maxima,
degenerate and fully masked chips between measured ones, box sums carried over odd and large
steps, chip areas whose statistics are not exact integers, the smallest and largest surfaces, and
points at the image's border."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (chip, radius x, radius y): remainders of the 16-row blocks, of the 32-row halves and of the 16
# columns of a lane quarter, both accumulator strides, every block height up to 64 px.
CASES = [(4, 1, 1), (8, 3, 2), (16, 8, 8), (16, 32, 32), (20, 17, 9), (32, 25, 25), (32, 16, 32),
         (32, 32, 15), (36, 29, 30), (48, 12, 26), (64, 25, 25), (64, 8, 32)]


def scene(seed):
    rng = np.random.default_rng(seed)
    ref = rng.integers(60, 200, (300, 301)).astype(np.uint8)
    k = np.ones(5) / 5
    for ax in (0, 1):
        ref = np.apply_along_axis(lambda v: np.convolve(v, k, "same"), ax, ref)
    ref = np.clip((ref - 128) * 3 + 128, 0, 255).astype(np.uint8)
    sec = np.roll(ref, (2, -3), (0, 1))
    ref[:, 190:] = 0           # windows that are zero, or partly so
    ref[150:230, 100:190] = 90  # flat windows, one grey level apart at one pixel
    ref[190, 140] = 91
    ref[:90, 100:190] = np.tile(ref[:9, 100:109], (10, 10))  # a repeated tile: equal maxima
    sec[40:110, 40:110] = 77   # degenerate chips
    valid = np.ones(ref.shape, bool)
    valid[180:290, 20:90] = False  # chips without a valid pixel
    return ref, sec, valid


@pytest.mark.parametrize("chip,rx,ry", CASES)
@pytest.mark.parametrize("measure", ["zncc", "ncc"])
@pytest.mark.parametrize("step", [1, 7, 24])
def test_identical_to_direct(ar, gpu_lib, chip, rx, ry, measure, step):
    ref, sec, valid = scene(chip + step)
    # Columns of points `step` rows apart (carried sums), then scattered ones.
    rng = np.random.default_rng(step)
    ys = np.arange(-5, 306, step)[:80]
    xs = np.array([12, 62, 75, 121, 150, 185, 230, 296])
    x = np.concatenate([np.repeat(xs, ys.size), rng.uniform(-5, 306, 60)]).astype(float)
    y = np.concatenate([np.tile(ys, xs.size), rng.uniform(-5, 306, 60)]).astype(float)
    pts = ar.pointset(x, y, chip_size=chip, search_radius_x=rx, search_radius_y=ry,
                      dx_prior=rng.integers(-2, 3, x.size).astype(float))
    pair = ar.ImagePair(ref, sec, None, valid)
    ctx = ar._lib.default_context()
    got = {}
    try:
        for up in (1, 8):
            p = ar.params(preprocess="none", quantize="none", similarity=measure,
                          subpixel="none" if up == 1 else ar.PyramidRefine(up))
            for kernel in (2, 0):
                ctx.set_option(ar._lib.AR_OPT_UINT8_KERNEL, kernel)
                got[up, kernel] = ar.track(pair, pts, p, ctx=ctx)
    finally:
        ctx.set_option(ar._lib.AR_OPT_UINT8_KERNEL, -1)
    for up in (1, 8):
        for name in ("dx", "dy", "correlation"):
            a, b = (getattr(got[up, k], name).view(np.uint32) for k in (2, 0))
            assert np.array_equal(a, b), (up, name, np.flatnonzero(a != b)[:5])
        assert np.array_equal(got[up, 2].searched, got[up, 0].searched)
    assert got[8, 2].searched.any() and not got[8, 2].searched.all()
