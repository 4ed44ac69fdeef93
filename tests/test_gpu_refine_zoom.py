"""k_refine's zoom search against the full Float32 cascade on bare 5 x 5 patches: identical value
and row-major-first position at every factor, for peaks anywhere in the patch and for patches
whose candidates never shrink to one tile (flat, tied, several peaks, rough, non-finite)."""

import numpy as np
import pytest

from test_refine_search import pyrup_fast

pytestmark = pytest.mark.gpu


def patches(kind, rng, count):
    i, j = np.mgrid[0:5, 0:5]
    out = np.empty((count, 5, 5), np.float32)
    for k in range(count):
        if kind == "peak":  # a smooth peak, also beyond the patch's edges
            r, c, w = rng.uniform(-1, 5), rng.uniform(-1, 5), rng.uniform(0.7, 6)
            p = rng.uniform(0.05, 1) * np.exp(-((i - r) ** 2 + (j - c) ** 2) / (2 * w * w))
            p = p + rng.choice([0.0, 0.01, 0.1]) * rng.standard_normal((5, 5)) - rng.uniform(0, 0.5)
        elif kind == "rough":
            p = rng.standard_normal((5, 5))
        elif kind == "flat":  # constant, or constant but for a few last bits
            p = np.full((5, 5), rng.uniform(-1, 1), np.float32)
            p = np.nextafter(p, p + rng.integers(-1, 2, (5, 5)).astype(np.float32) * (k % 2))
        elif kind == "tied":  # several equal maxima
            p = rng.integers(0, 2, (5, 5)).astype(float)
        elif kind == "ridge":
            p = 1 - 1e-3 * (i * np.cos(k) + j * np.sin(k) - 2) ** 2
        else:  # non-finite and huge values
            p = rng.standard_normal((5, 5))
            bad = [np.nan, np.inf, -np.inf, 3e38, -3e38][k % 5]
            p[rng.random((5, 5)) < rng.choice([0.05, 0.5, 1.0])] = bad
        out[k] = p
    return out


@pytest.mark.parametrize("up", [2, 4, 8, 16, 64, 128])
@pytest.mark.parametrize("kind", ["peak", "rough", "flat", "tied", "ridge", "nonfinite"])
def test_zoom_matches_cascade(ar, gpu_lib, up, kind):
    rng = np.random.default_rng(up)
    P = patches(kind, rng, 400 if kind == "peak" else 40)
    row, col, val = ar.refine_patches(P, up)
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
                assert np.isnan(val[k]) or val[k] == flat[0], k
