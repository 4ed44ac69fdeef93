"""The box-tile filters and the pair masks at the edges of their tiles and runs, against the oracle.

Window sums come in runs of eight outputs, from shared parts once the window is eight wide, on tiles
of 32 x 64 pixels; an even window is a wider one clamped to the image. Float32 imagery that holds whole numbers sums
exactly in FP64 in any order, so the highpass is bit-identical. Wallis deviations are squares of
Float32 values whose FP64 sums may round apart from the oracle's in the last place: one Float32 ulp
of the deviation, 1e-6 of the value and a margin. A flat stretch has a deviation of exactly zero and
stays invalid, however large its neighbourhood's values are.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _image(rng, shape):
    a = rng.integers(0, 4096, shape).astype(np.float32)
    a[: shape[0] // 3, shape[1] // 2:] = 1000.0
    m = rng.random(shape) > 0.002
    return a, m


def _both(ar, O, a, m, p, *args):
    b, k = np.asfortranarray(a[::-1]), np.asfortranarray(m[::-1])
    r, s, rm, sm = ar.prepare(ar.ImagePair(a, b, m, k), p).download()
    for img, mask, got, gm in ((a, m, r, rm), (b, k, s, sm)):
        want, wm = O.prepare(img, mask, *args)
        assert np.array_equal(gm, wm)
        yield got, want


@pytest.mark.parametrize("width,shape", [(3, (33, 65)), (7, (64, 128)), (9, (31, 63)), (9, (97, 130)),
                                         (21, (129, 191)), (21, (8, 300)), (21, (301, 6)),
                                         (63, (150, 140)), (63, (70, 60))])
def test_highpass_of_floats_exact(ar, O, gpu_lib, width, shape):
    a, m = _image(np.random.default_rng(width), shape)
    p = ar.params(quantize="none", filter_width=width)
    for got, want in _both(ar, O, a, m, p, "highpass", width, 0.0, "none"):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("width,shape", [(5, (33, 65)), (9, (63, 129)), (21, (129, 191)),
                                         (63, (150, 140))])
def test_wallis_flat_and_textured(ar, O, gpu_lib, width, shape):
    a, m = _image(np.random.default_rng(width), shape)
    p = ar.params(preprocess=ar.Wallis(width=width, min_std=0.0), quantize="none")
    for got, want in _both(ar, O, a, m, p, "wallis", width, 0.0, "none"):
        assert np.all(np.abs(got - want) <= 1e-6 * np.maximum(1.0, np.abs(want)))


@pytest.mark.parametrize("shape", [(16, 16), (37, 29), (15, 1), (3, 5), (255, 257)])
@pytest.mark.parametrize("dtype", [np.uint8, np.float32])
@pytest.mark.parametrize("given", [(False, False), (True, False), (False, True), (True, True)])
def test_pair_masks_of_any_size(ar, gpu_lib, shape, dtype, given):
    rng = np.random.default_rng(shape[0])
    a = rng.integers(1, 200, shape).astype(dtype)
    b = rng.integers(1, 200, shape).astype(dtype)
    if dtype is np.float32:
        a.flat[::7] = np.nan
        b.flat[3::11] = np.inf
    ms = [rng.random(shape) > 0.3 if g else None for g in given]
    p = ar.params(preprocess="none", quantize="none")
    _, _, rm, sm = ar.prepare(ar.ImagePair(a, b, *ms), p).download()
    for got, img, m in ((rm, a, ms[0]), (sm, b, ms[1])):
        assert np.array_equal(got, np.isfinite(img) if m is None else m)
