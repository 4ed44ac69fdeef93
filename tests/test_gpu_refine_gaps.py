"""k_refine on patches with NaN, of zeros and of noise, against the full Float32 cascade: identical value and
row-major-first position at every factor. NaN at each of the 25 places, whole rows and columns of them,
few values left, beside smooth peaks, rough and tied values; zeros of either sign."""

import numpy as np
import pytest

from test_refine_search import pyrup_fast

pytestmark = pytest.mark.gpu


def patches(kind, rng):
    i, j = np.mgrid[0:5, 0:5]

    def base(k):
        if k % 3 == 0:
            r, c, w = rng.uniform(0, 4), rng.uniform(0, 4), rng.uniform(0.7, 4)
            return np.exp(-((i - r) ** 2 + (j - c) ** 2) / (2 * w * w)) - rng.uniform(0, 0.5)
        return rng.standard_normal((5, 5)) if k % 3 == 1 else rng.integers(0, 2, (5, 5)).astype(float)

    out = []
    if kind == "one":
        for at in range(25):
            for k in range(3):
                p = base(k)
                p.flat[at] = np.nan
                out.append(p)
    elif kind == "many":
        for k in range(60):
            p = base(k)
            p[rng.random((5, 5)) < rng.choice([0.1, 0.4, 0.8])] = np.nan
            if k % 4 == 0:
                p[rng.integers(5)] = np.nan
            if k % 4 == 1:
                p[:, rng.integers(5)] = np.nan
            out.append(p)
        out.append(np.full((5, 5), np.nan))
    elif kind == "rough":  # boxes that do not shrink; infinite and huge values
        out = [rng.standard_normal((5, 5)) for _ in range(40)]
        out += [np.where(rng.random((5, 5)) < 0.1, bad, base(1)) for bad in (np.inf, -np.inf, 3e38)]
    else:
        out = [np.zeros((5, 5)), -np.zeros((5, 5)), np.where((i + j) % 2, 0.0, -0.0)]
        out += [np.where((i == r) & (j == c), v, 0.0) for r, c in ((0, 0), (2, 2), (4, 4), (0, 3)) for v in (1e-45, -1.0)]
    return np.array(out, np.float32)


@pytest.mark.parametrize("up", [2, 4, 8, 16, 64, 128])
@pytest.mark.parametrize("kind", ["one", "many", "zeros", "rough"])
@pytest.mark.parametrize("count", [1, 2, 592, 593])
def test_matches_cascade(ar, gpu_lib, up, kind, count):
    """Up to 592 patches a block of four warps takes each, beyond a warp does."""
    P = patches(kind, np.random.default_rng(up))
    row, col, val = (v.reshape(-1) for v in ar.refine_patches(np.resize(P, (count, 5, 5)), up))
    P = P[:count]
    with np.errstate(all="ignore"):
        for k, p in enumerate(P):
            s = p
            while s.shape[0] < 5 * up:
                s = pyrup_fast(s)
            flat = s.reshape(-1)
            good = flat[flat > -np.inf]
            at = int(np.flatnonzero(flat == good.max())[0]) if good.size else 0
            assert (row[k], col[k]) == divmod(at, 5 * up), k
            if good.size:
                assert val[k] == flat[at], k
            else:
                assert np.isnan(val[k]), k
