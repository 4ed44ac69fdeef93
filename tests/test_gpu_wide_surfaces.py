"""k_corr_tc on surfaces beyond 64 x 64 at the edges of its layouts, bit-identical to the CUDA-core
kernel (exact integer numerators and sums, the same FP64 normalisation).

Layouts: two blocks an SM with the whole chip operand (16, 34), with the operand in chunks (32, 44),
one block with the reciprocal roots kept (32, 60) and without (48, 50); M = 64 products on tall narrow
surfaces; stripes and 16-row reads with remainders. The scene has flat and repeating stretches, where
the largest estimate does not stand out and the values near it are compared exactly.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(16, 34, 33), (16, 48, 48), (20, 41, 37), (32, 44, 44), (32, 47, 35), (32, 60, 50),
         (48, 50, 50), (12, 10, 33), (24, 32, 60), (64, 20, 40), (4, 33, 2), (16, 56, 36)]


def scene(seed):
    rng = np.random.default_rng(seed)
    ref = rng.integers(0, 256, (420, 400)).astype(np.uint8)
    sec = np.roll(ref, (-3, 2), (0, 1))
    ref[:, 280:] = np.tile(rng.integers(0, 256, (8, 8)).astype(np.uint8), (53, 15))[:420]
    sec[:, 280:] = ref[:, 280:]
    ref[100:230, 20:150] = 0
    sec[300:360, 40:200] = 77
    valid = np.ones(ref.shape, bool)
    valid[180:260, 200:260] = False
    return ref, sec, valid


@pytest.mark.parametrize("chip,rx,ry", CASES)
@pytest.mark.parametrize("measure", ["zncc", "ncc"])
@pytest.mark.parametrize("up", [1, 8])
def test_identical_to_direct(ar, gpu_lib, chip, rx, ry, measure, up):
    ref, sec, valid = scene(chip + rx)
    rng = np.random.default_rng(ry)
    # Columns of points a few rows apart (carried sums), then scattered ones of mixed radii.
    xs, ys = np.array([60, 110, 160, 215, 262, 310, 340]), np.arange(40, 380, 9)
    x = np.concatenate([np.repeat(xs, ys.size), rng.uniform(-5, 405, 80)]).astype(float)
    y = np.concatenate([np.tile(ys, xs.size), rng.uniform(-5, 425, 80)]).astype(float)
    n = xs.size * ys.size
    rxs, rys = np.full(x.size, rx), np.full(x.size, ry)
    rxs[n:] = rng.integers(1, rx + 1, 80)
    rys[n:] = rng.integers(1, ry + 1, 80)
    pts = ar.pointset(x, y, chip_size=chip, search_radius_x=rxs, search_radius_y=rys)
    pair = ar.ImagePair(ref, sec, None, valid)
    p = ar.params(preprocess="none", quantize="none", similarity=measure,
                  subpixel="none" if up == 1 else ar.PyramidRefine(up))
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
        assert np.array_equal(a, b), (name, np.flatnonzero(a != b)[:5])
    assert np.array_equal(got[1].searched, got[0].searched)
    assert np.count_nonzero(~np.isnan(got[1].dx)) > x.size // 2
