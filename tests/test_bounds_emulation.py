"""Host emulations of bounds and roundings that kernels rely on:

* a product with the rounded reciprocal and one correction (a remainder and a multiply-add) is the rounded
  quotient, for every sum the highpass of integer imagery can meet (Float32) and for sums over every window
  area of the box filters (FP64);
* k_refine's zoom: the final samples of a cell of any level are below its largest corner plus the bound made of
  second differences, and a node's final sample is at least the node less the bound;
* the Float32 estimates of k_corr_tc2 and k_corr_tc lie within their one bound a point of the exact values.
"""

from fractions import Fraction

import numpy as np
import pytest

F32, LD = np.float32, np.longdouble


@pytest.mark.parametrize("W", [3, 5, 7, 9])
@pytest.mark.parametrize("bias", [0, 32768])
def test_corrected_quotient_of_every_sum(W, bias):
    n = W * W
    a = np.arange(0, n * 65535 + 1, dtype=np.int64) - bias * n
    af, inv = a.astype(F32), F32(1) / F32(n)
    assert np.array_equal(af.astype(np.int64), a)
    q = af * inv
    rem = (af.astype(LD) - q.astype(LD) * n).astype(F32)  # exact: a multiple of q's last place, a few of them
    got = (q.astype(LD) + rem.astype(LD) * LD(inv)).astype(F32)
    assert np.array_equal(got, (a.astype(np.float64) / n).astype(F32))


def test_corrected_quotient_of_window_areas():
    rng = np.random.default_rng(0)
    for n in sorted({wx * wy for wx in range(1, 64) for wy in range(1, 64)})[::9]:
        inv = 1.0 / float(n)
        for s in rng.integers(1 << 52, 1 << 53, 60):
            s = float(s)
            q = s * inv
            rem = float(Fraction(s) - Fraction(q) * n)  # a multiply-add: one rounding, here none
            assert Fraction(rem) == Fraction(s) - Fraction(q) * n
            assert float(Fraction(q) + Fraction(rem) * Fraction(inv)) == s / n, (n, s)


def pyrup(s):
    def step(v):  # along axis 0
        n = v.shape[0]
        m, q = np.r_[min(1, n - 1), 0:n - 1], np.r_[1:n, n - 1]
        out = np.empty((2 * n,) + v.shape[1:])
        out[0::2] = 0.75 * v + 0.125 * (v[m] + v[q])
        out[1::2] = 0.5 * (v + v[q])
        return out
    return step(step(s).T).T


def second(v):
    n = v.shape[0]
    m, q = np.r_[1, 0:n - 1], np.r_[1:n, n - 1]
    return np.abs(v[m] + v[q] - 2 * v).max()


@pytest.mark.parametrize("kind", ["rough", "peak", "tied"])
def test_zoom_bound(kind):
    rng = np.random.default_rng(1)
    i, j = np.mgrid[0:5, 0:5]
    for _ in range(60):
        if kind == "rough":
            p = rng.standard_normal((5, 5))
        elif kind == "peak":
            p = np.exp(-((i - rng.uniform(0, 4)) ** 2 + (j - rng.uniform(0, 4)) ** 2) / rng.uniform(1, 8))
        else:
            p = rng.integers(0, 2, (5, 5)).astype(float)
        levels = [p]
        while levels[-1].shape[0] < 160:
            levels.append(pyrup(levels[-1]))
        fin = levels[-1]
        e1 = (second(levels[1]) + second(levels[1].T)) / 6
        assert e1 <= (second(p) + second(p.T)) / 24 + 1e-12
        for l in range(1, 5):
            v, e = levels[l], e1 * 4.0 ** (1 - l) + 1e-9
            f = 1 << (5 - l)
            assert (fin[::f, ::f] >= v - e).all()
            hi = v.copy()  # the largest corner of the cell from node (r, c) on (the last node again beyond)
            up = np.pad(v, ((0, 1), (0, 1)), mode="edge")
            for a in (0, 1):
                for b in (0, 1):
                    hi = np.maximum(hi, up[a:a + v.shape[0], b:b + v.shape[1]])
            cells = fin.reshape(v.shape[0], f, v.shape[1], f).max(axis=(1, 3))
            assert (cells <= hi + e).all()


@pytest.mark.parametrize("measure", ["zncc", "ncc"])
@pytest.mark.parametrize("ch,cw", [(16, 16), (32, 32), (20, 12), (100, 100)])
def test_estimates_within_their_bound(measure, ch, cw):
    rng = np.random.default_rng(ch + cw)
    nn, nnf = ch * cw, F32(ch * cw)
    u24 = F32(6.02e-08)
    made = 0
    for t in range(300):
        lo = rng.integers(0, 200)
        spread = int(rng.choice([2, 8, 60, 255 - lo]))
        C = rng.integers(lo, min(lo + spread, 255) + 1, nn).astype(np.int64)
        w0 = rng.integers(0, 240)
        W = np.clip(w0 + rng.integers(0, int(rng.choice([2, 5, 40, 200])), nn), 0, 255).astype(np.int64)
        if t % 3 == 0:
            W = np.clip(C + rng.integers(-3, 4, nn), 0, 255)
        D, s1, s2 = int((C * W).sum()), int(W.sum()), int((W * W).sum())
        cs, c2 = int(C.sum()), int((C * C).sum())
        sq = (nn * c2 - cs * cs) / nn
        vx_exact = s2 if measure == "ncc" else nn * s2 - s1 * s1
        if sq == 0 or s2 == 0:
            continue
        # As the kernels: every operation rounded to Float32, D and s2 converted, s1 and cs exact.
        Df, s1f, s2f, csf = F32(D), F32(s1), F32(s2), F32(cs)
        q = s1f * s1f
        vx = s2f if measure == "ncc" else F32(np.float64(nnf) * np.float64(s2f) - np.float64(q))
        if measure == "zncc" and F32(np.float64(nnf) * np.float64(s2f) + np.float64(q)) > F32(2048) * vx:
            continue  # evaluated exactly
        r = F32(1 / np.sqrt(np.float64(vx))) * F32(1 + 2 * 2.0 ** -23 * rng.uniform(-1, 1))  # 2 ulp
        nx = F32(np.float64(nnf) * np.float64(Df) - np.float64(csf * s1f))
        est = nx * r
        kz, kc = np.sqrt(F32(sq) * nnf), np.sqrt(nnf * F32(c2))
        bu = (u24 * np.sqrt(nnf) * (F32(20) * kz + F32(5) * kc) if measure == "ncc"
              else u24 * (F32(3400) * kz + F32(160) * kc))
        value = (nn * D - cs * s1) / np.sqrt(np.float64(vx_exact))
        assert abs(float(est) - value) <= float(bu)
        made += 1
    assert made > 60
