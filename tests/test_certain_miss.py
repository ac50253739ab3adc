"""The mathematics of the single-precision rule that drops a leaf's triangles before the double test
(certain_miss in bf200_triangle.cuh), restated in numpy: whenever it applies, two exact edge functions have
opposite signs, which the double test answers with a miss. test_device_rules.py checks the header's own
code."""
from fractions import Fraction

import numpy as np
import pytest

F, D = np.float32, np.float64


def fma(a, b, c):
    """Products of two floats are exact in double; the sum rounds once there and once to float."""
    return (a.astype(D) * b.astype(D) + c.astype(D)).astype(F)


def certain_miss(v, o, d):
    p = [(v[k] - o).astype(F) for k in range(3)]
    f = [(v[2] - v[1]).astype(F), (v[0] - v[2]).astype(F), (v[1] - v[0]).astype(F)]

    def edge(p, f):
        c = [fma(p[:, a], f[:, b], -(p[:, b] * f[:, a]).astype(F)) for a, b in ((1, 2), (2, 0), (0, 1))]
        return fma(d[:, 0], c[0], fma(d[:, 1], c[1], (d[:, 2] * c[2]).astype(F)))

    d_sum = (np.abs(d[:, 0]) + np.abs(d[:, 1]) + np.abs(d[:, 2])).astype(F)
    pm = np.abs(np.concatenate(p, axis=1)).max(axis=1)
    fm = np.abs(np.concatenate(f, axis=1)).max(axis=1)
    bound = np.fmax(F(4.0) * pm * fm * d_sum * F(5.0 * 5.9604645e-8), F(1e-30) * (F(1.0) + d_sum)).astype(F)
    e = np.stack([edge(p[1], f[0]), edge(p[2], f[1]), edge(p[0], f[2])])
    return (e > bound).any(axis=0) & (e < -bound).any(axis=0)


def exact_signs(v, o, d):
    q = [[Fraction(float(v[k][a])) - Fraction(float(o[a])) for a in range(3)] for k in range(3)]
    r = [Fraction(float(x)) for x in d]
    signs = []
    for i, j in ((1, 2), (2, 0), (0, 1)):
        p, s = q[i], q[j]
        value = sum(r[a] * (p[(a + 1) % 3] * s[(a + 2) % 3] - p[(a + 2) % 3] * s[(a + 1) % 3]) for a in range(3))
        signs.append((value > 0) - (value < 0))
    return signs


@pytest.mark.parametrize("distance", [1e-3, 1.0, 30.0, 1e4, 1e12, 1e20])
@pytest.mark.parametrize("size", [1e-12, 1e-3, 1.0, 1e18, 1e20])
def test_certain_misses_are_misses(distance, size):
    rng = np.random.default_rng(int(1000 * np.log10(distance)) % 977 + abs(int(np.log10(size))))
    n = 3000
    v = [(rng.normal(size=(n, 3)) * size).astype(F) for _ in range(3)]
    w = rng.dirichlet((1.0, 1.0, 1.0), n)
    w[::2, 0] = rng.normal(size=len(w[::2])) * 10.0 ** rng.uniform(-9.0, 0.0, len(w[::2]))  # near an edge
    target = sum(w[:, k:k + 1] * v[k] for k in range(3)) / w.sum(axis=1, keepdims=True)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(F)
    o = (target - distance * d).astype(F)
    with np.errstate(all="ignore"):
        certain = certain_miss(v, o, d)
    for k in np.nonzero(certain)[0]:
        signs = exact_signs([x[k] for x in v], o[k], d[k])
        assert 1 in signs and -1 in signs, k
    if size / distance >= 1e-3 and 1e-10 < size < 1e10:  # near enough for the rule to decide anything
        assert certain.any()
