"""Raw Float32 windows with NaN or infinite pixels, against sums kept as the general kernel keeps them.

The FP64 running sums behind a window's variance start afresh every sixteen surface columns and run
on down the rows, so a pixel that is not finite at window row r, column c leaves no number in any value
(i, j) with i + ch > r whose run of sixteen columns starts at or left of c, j + cw > c: those values are
0. (The oracle's summed-area tables do the same without the runs: up to sixteen surface columns the
expected surface is the oracle's own.) Every other value is that of the window without those
pixels; the FP32 products of two chip columns keep it within 1e-5 of the FP64 one. Chips of whole sixteens:
the zero rows below other chips meet the pixel in the products.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (chip, radius x, radius y): within one run of columns, across runs, one and two row tiles.
CASES = [(16, 8, 8), (16, 4, 20), (32, 8, 25), (32, 25, 25), (16, 20, 9), (48, 32, 32), (32, 32, 30)]


def window(chip, rx, ry, bad, seed):
    rng = np.random.default_rng(seed)
    w = rng.standard_normal((chip + 2 * ry - 1, chip + 2 * rx - 1)).astype(np.float32) * 50 + 7
    c = w[ry:ry + chip, rx - 1:rx - 1 + chip] + rng.standard_normal((chip, chip)).astype(np.float32)
    at = [(rng.integers(w.shape[0] // 3, w.shape[0]), rng.integers(0, w.shape[1])) for _ in range(2)]
    if seed % 3 == 0:
        at = [(w.shape[0] // 2, w.shape[1] // 2), (w.shape[0] - 1, 0)]
    clean = w.copy()
    for k, (r, q) in enumerate(at):
        w[r, q] = bad if k == 0 else np.nan
        clean[r, q] = 0
    return w, clean, c, at


def without_variance(nr, nc, ch, cw, at, tile_rows):
    z = np.zeros((nr, nc), bool)
    i, j = np.mgrid[0:nr, 0:nc]
    for r, c in at:
        # A row tile's sums start at its first row.
        z |= (i + ch > r) & (i // tile_rows * tile_rows <= r) & (j // 16 * 16 <= c) & (j + cw > c)
    return z


@pytest.mark.parametrize("chip,rx,ry", CASES)
@pytest.mark.parametrize("bad,measure", [(np.nan, "zncc"), (np.inf, "zncc"), (-np.inf, "zncc"), (np.nan, "ncc")])
@pytest.mark.parametrize("seed", [1, 3])
def test_surface(ar, O, gpu_lib, chip, rx, ry, bad, measure, seed):
    w, clean, c, at = window(chip, rx, ry, bad, seed)
    nr, nc = 2 * ry, 2 * rx
    # Groups of ten rows for each of 256 / nc threads a column (a block's tile).
    z = without_variance(nr, nc, chip, chip, at, min(-(-nr // 10), 256 // nc) * 10)
    want, _ = O.correlate(clean, c, (rx, ry), measure=measure)
    want = np.where(z, 0.0, want)
    got, degenerate = ar.correlate(w, c, (rx, ry), measure=ar.NCC() if measure == "ncc" else ar.ZNCC())
    assert not degenerate
    assert np.array_equal(got == 0, want == 0)
    assert np.abs(got - want).max() <= 1e-5
    if nc <= 16 and measure == "zncc":
        ref, _ = O.correlate(w, c, (rx, ry), measure=measure)
        assert np.array_equal(ref == 0, want == 0)


@pytest.mark.parametrize("angles", [None, (0.0,), (-3.0, 0.0, 2.0)])
@pytest.mark.parametrize("chip,rx,ry", [(16, 8, 8), (32, 8, 20), (16, 5, 30)])
def test_pass_over_an_image_with_gaps(ar, O, gpu_lib, angles, chip, rx, ry):
    """One run of columns and one row tile: the oracle's tables and the kernel's lose the same values, so
    the peaks are the oracle's (noise imagery: no two values within the FP32 products' 1e-5)."""
    rng = np.random.default_rng(chip + ry)
    a = rng.standard_normal((240, 250)).astype(np.float32)
    b = (np.roll(a, (3, -2), (0, 1)) + 0.05 * rng.standard_normal(a.shape)).astype(np.float32)
    gaps = rng.random(a.shape) < 4e-4
    a[gaps] = np.where(rng.random(gaps.sum()) < 0.6, np.nan, np.inf)
    ones = np.ones(a.shape, bool)
    n = 150
    pts = ar.pointset(rng.uniform(0, 250, n), rng.uniform(0, 240, n), chip_size=chip, search_radius_x=rx,
                      search_radius_y=ry, dx_prior=rng.integers(-2, 3, n).astype(float), dy_prior=0.0)
    p = ar.params(preprocess="none", quantize="none", subpixel="none", rotation=angles)
    got = ar.track(ar.ImagePair(a, b, ones, ones), pts, p)
    want = O.track(a, b, {f: getattr(pts, f) for f in ar.points.FIELDS}, upsampling=1,
                   angles=None if angles is None else np.array(angles))
    assert np.array_equal(got.searched, want[3])
    assert np.array_equal(got.dx, want[0], equal_nan=True) and np.array_equal(got.dy, want[1], equal_nan=True)
    m = ~np.isnan(want[0])
    assert np.abs(got.correlation[m] - want[2][m]).max() <= 1e-5
    assert 5 < np.count_nonzero(want[2][m] < 0.5) < m.sum() - 5  # both kinds of points are there
