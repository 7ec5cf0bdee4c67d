"""The margins of the double-precision count pass (float_test in csrc/radius_graph.cu), restated in numpy: a pair decided by its
float distance must be decided as the double test decides it.  The formula is restated here, the kernel's own outputs are
compared with the double-precision oracle in test_radius_graph_gpu.py."""

import numpy as np
import pytest

U = 2.0 ** -24
EPS = float(np.float32(1e-8))


def _margin(t2, X):
    t = np.sqrt(t2)
    eta = 2.0 * U * X
    e = eta + U * t
    return 2.0 * (3.5 * t * eta + 6.0 * U * t2 + 3.0 * e * e)


def _outward(v, up):
    f = np.float32(v)
    if up and float(f) < v:
        f = np.nextafter(f, np.float32(np.inf))
    if not up and float(f) > v:
        f = np.nextafter(f, np.float32(-np.inf))
    return f


def _fma32(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(np.float32)


@pytest.mark.parametrize("X", [10.0, 470.0, 1.0e4, 1.0e6, 1.0e8])
@pytest.mark.parametrize("r", [0.5, 5.0, 12.0])
def test_decided_pairs_agree_with_the_double_test(X, r):
    rng = np.random.default_rng(5)
    n = 200_000
    a = rng.random((n, 3)) * X
    dirs = rng.normal(size=(n, 3))
    dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
    scale = np.where(rng.random(n) < 0.5, r, 1.0e-4) * (1.0 + rng.normal(size=n) * 10.0 ** rng.uniform(-12, 0.5, n))
    b = np.clip(a + dirs * scale[:, None], 0.0, X)
    b[:100] = a[:100]
    d = a - b
    exact2 = (d * d).sum(axis=1)
    hit = (exact2 <= r * r) & (exact2 > EPS)
    fa, fb = a.astype(np.float32), b.astype(np.float32)
    f = fa - fb
    d32 = _fma32(f[:, 2], f[:, 2], _fma32(f[:, 0], f[:, 0], f[:, 1] * f[:, 1]))
    near, lo, hi = _outward(EPS + _margin(EPS, X), True), _outward(r * r - _margin(r * r, X), False), _outward(r * r + _margin(r * r, X), True)
    sure = (d32 <= lo) & (d32 > near)
    none = d32 > hi
    assert hit[sure].all() and not hit[none].any()
    if X <= 1.0e4:
        assert sure.any() and none.any()      # most pairs lie inside the margins by construction
    if 3.1 * (2.0 * U * X) ** 2 < EPS:        # equal floats lie inside the self-distance limit
        same = (fa == fb).all(axis=1)
        assert same[:100].all() and not hit[same].any()
