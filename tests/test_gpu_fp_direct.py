"""k_corr_fp (direct FP32 over one-tile surfaces, and turned chips) against the oracle where its
tiling can go wrong: row groups of ten and column pairs that fill the block, half of it, or a few
threads (the chip's columns then split over 2, 4 or 8 parts), surfaces just beyond one tile (the
general kernel), chip sides off the multiples of 16, windows at the border, zero and repeated
areas, NCC.

Integer peaks (no refinement): the correlation is within 1e-5 of the FP64 one (FP32 products of two
chip columns, FP64 beyond), so the reported value is within 1e-5 of the oracle's maximum and the
displacement is the same wherever the oracle has no second value within 2e-5 of it; ties and
near-ties are left out by comparing displacements only where a one-pixel texture makes the margin
large (asserted to be most points).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (chip, radius x, radius y)
CASES = [(4, 1, 1), (8, 2, 5), (16, 6, 7), (20, 10, 10), (24, 16, 11), (32, 25, 25), (32, 3, 32),
         (48, 32, 20), (12, 32, 32), (32, 28, 45), (36, 20, 15), (60, 11, 6)]


def scene(dtype, seed):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((230, 231))
    a = a + 0.3 * np.roll(a, 1, 0) + 0.3 * np.roll(a, 1, 1)
    b = np.roll(a, (2, -3), (0, 1)) + 0.02 * rng.standard_normal(a.shape)
    if dtype == np.float32:
        a, b = (v.astype(dtype) for v in (500 * a, 500 * b))
    elif dtype == np.int16:
        a, b = (np.round(500 * v).astype(dtype) for v in (a, b))
    else:
        hi = 255 if dtype == np.uint8 else 65535
        a, b = (np.clip(np.round(hi * (0.5 + 0.12 * v)), 0, hi).astype(dtype) for v in (a, b))
    a = a.copy()
    a[150:, 150:] = 0          # windows of zeros
    b[20:60, 150:200] = b[20, 150]  # degenerate chips
    valid = np.ones(a.shape, bool)
    valid[150:220, 10:90] = False
    return a, b, valid


def points(ar, chip, rx, ry, seed):
    rng = np.random.default_rng(seed)
    n = 260
    x, y = rng.uniform(-8, 240, n), rng.uniform(-8, 240, n)
    return ar.pointset(x, y, chip_size=chip, search_radius_x=rx, search_radius_y=ry,
                       dx_prior=rng.integers(-2, 3, n).astype(float), dy_prior=0.0)


def compare(ar, O, dtype, chip, rx, ry, measure, angles):
    a, b, valid = scene(dtype, chip + rx)
    pts = points(ar, chip, rx, ry, ry)
    p = ar.params(preprocess="none", quantize="none", similarity=measure, subpixel="none",
                  rotation=angles)
    g = ar.track(ar.ImagePair(a, b, None, valid), pts, p)
    fields = {n: getattr(pts, n) for n in ar.points.FIELDS}
    w = O.track(a, b, fields, upsampling=1, measure=measure, secondary_valid=valid,
                angles=None if angles is None else np.array(angles))
    assert np.array_equal(g.searched, w[3])
    assert np.array_equal(np.isnan(g.dx), np.isnan(w[0]))
    m = ~np.isnan(w[0])
    assert m.sum() > 40
    assert np.abs(g.correlation[m] - w[2][m]).max() <= 1e-5
    # A chip of 8 px and up whose true position lies in the window: a peak far above the rest.
    sharp = m & (w[2] > 0.9)
    if chip >= 8 and rx > 5 and ry > 5 and measure == "zncc":
        assert sharp.sum() > m.sum() // 4
        assert np.array_equal(g.dx[sharp], w[0][sharp]) and np.array_equal(g.dy[sharp], w[1][sharp])


@pytest.mark.parametrize("dtype", [np.float32, np.uint16, np.int16])
@pytest.mark.parametrize("chip,rx,ry", CASES)
@pytest.mark.parametrize("measure", ["zncc", "ncc"])
def test_direct(ar, O, gpu_lib, dtype, chip, rx, ry, measure):
    compare(ar, O, dtype, chip, rx, ry, measure, None)


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.float32])
@pytest.mark.parametrize("chip,rx,ry", CASES)
def test_turned(ar, O, gpu_lib, dtype, chip, rx, ry):
    compare(ar, O, dtype, chip, rx, ry, "zncc", (-4.0, 0.0, 3.0))
