"""The box-tile filters' two tile shapes (32 x 32 with runs of four sums for windows below eight and small images,
32 x 64 with runs of eight) at the edges of their tiles and runs, against the oracle: whole-number Float32 imagery sums exactly in FP64, so the highpass is
bit-identical; Wallis within one Float32 ulp of its deviation (1e-6 with a margin). An image smaller than
the filter clamps the window, to even widths as well."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(32, 32), (33, 31), (31, 33), (64, 65), (97, 40), (1, 40), (40, 2), (5, 4), (6, 70), (3, 3)]


def _image(rng, shape):
    a = rng.integers(0, 4096, shape).astype(np.float32)
    m = rng.random(shape) > 0.02
    return a, m


NARROW = [(w, s) for w in (3, 5, 7, 9, 21, 63) for s in SHAPES] + [(3, (650, 541)), (7, (577, 545))]
WIDE = [(9, (577, 545)), (21, (1201, 290)), (63, (640, 513))]  # more than 296 narrow tiles


@pytest.mark.parametrize("width,shape", NARROW + WIDE)
@pytest.mark.parametrize("filt", ["highpass", "wallis"])
def test_tile_shapes(ar, O, gpu_lib, width, shape, filt):
    rng = np.random.default_rng(width * 100 + shape[0])
    a, m = _image(rng, shape)
    b, k = _image(rng, shape)
    pre = ar.Highpass(width) if filt == "highpass" else ar.Wallis(width=width, min_std=0.0)
    r, s, rm, sm = ar.prepare(ar.ImagePair(a, b, m, k), ar.params(preprocess=pre, quantize="none")).download()
    for img, mask, got, gm in ((a, m, r, rm), (b, k, s, sm)):
        want, wm = O.prepare(img, mask, filt, width, 0.0, "none")
        assert np.array_equal(gm, wm)
        if filt == "highpass":
            assert np.array_equal(got, want)
        else:
            assert np.all(np.abs(got - want) <= 1e-6 * np.maximum(1.0, np.abs(want)))
