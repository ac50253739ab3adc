"""The device headers' own product, MIS and stepping rules and their triangle test, compiled for the host
(tests/device_rules.cpp): operations round there as on the device, so what holds here holds in the kernels."""
import ctypes as C
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from test_certain_miss import exact_signs
from test_factor_products import F, MAX_FLOAT, MIN_NORMAL, factors

CUDA_INCLUDE = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def rules(repo_root, tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are not available")
    library = tmp_path_factory.mktemp("rules") / "device_rules.so"
    source = os.path.join(repo_root, "blackframe-renderer_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", f"-I{CUDA_INCLUDE}",
                    f"-I{source}", "-o", str(library), os.path.join(repo_root, "tests", "device_rules.cpp")],
                   check=True)
    return C.CDLL(str(library))


def pointer(array):
    return array.ctypes.data_as(C.c_void_p)


def products(rules, num, den):
    """(direct, whether it applies, quotient form, ratio form) of columns of factors."""
    num, den = np.ascontiguousarray(num, F), np.ascontiguousarray(den, F)
    n = num.shape[1]
    direct, quotient, ratio = (np.zeros(n, F) for _ in range(3))
    applies = np.zeros(n, np.uint8)
    assert rules.rule_products(len(num), len(den), pointer(num), pointer(den), C.c_uint64(n), pointer(direct),
                               pointer(applies), pointer(quotient), pointer(ratio)) == 0
    return direct, applies != 0, quotient, ratio


def same_bits(a, b):
    return np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("counts", [(2, 1), (3, 1), (4, 1), (2, 2), (4, 3), (5, 2), (7, 2), (7, 4)])
def test_direct_products_equal_both_split_forms(rules, counts):
    rng = np.random.default_rng(23 * counts[0] + counts[1])
    direct, applies, quotient, ratio = products(rules, factors(rng, counts[0], 100_000), factors(rng, counts[1], 100_000))
    assert 0.05 < applies.mean() < 1.0
    assert same_bits(direct[applies], quotient[applies]) and same_bits(direct[applies], ratio[applies])


@pytest.mark.parametrize("by_quotient", [False, True])
def test_partial_products_beside_the_smallest_normal_number(rules, by_quotient):
    """A partial result just below the normal range may round up to its smallest number, losing the bit that
    the split forms keep: (1 - 2^-24) 2^-60 times 2^-66, then times 3."""
    rng = np.random.default_rng(41 + by_quotient)
    n = 50_000
    mantissa = (1.0 + rng.integers(-40, 40, n) * 2.0 ** -24).astype(F)
    other = np.where(rng.random(n) < 0.5, F(1.0), (1.0 + rng.integers(-4, 4, n) * 2.0 ** -24).astype(F)).astype(F)
    shift = rng.integers(20, 90, n)
    a = np.ldexp(mantissa, -shift).astype(F)
    last = rng.uniform(1.0, 4.0, n).astype(F)
    a[0], other[0], last[0], shift[0] = np.ldexp(F(1.0 - 2.0 ** -24), -60), 1.0, 3.0, 60
    if by_quotient:  # the small partial result comes from a division, and a later one brings it back
        num, den = [a, np.ones(n, F)], [np.ldexp(other, 126 - shift), (1.0 / last).astype(F)]
    else:
        num, den = [a, np.ldexp(other, shift - 126), last], [np.ones(n, F)]
    direct, applies, quotient, ratio = products(rules, num, den)
    assert same_bits(direct[applies], quotient[applies]) and same_bits(direct[applies], ratio[applies])
    assert 0.1 < applies.mean() < 0.9


def test_plain_products_of_two_equal_the_split_form(rules):
    rng = np.random.default_rng(7)
    a, b = factors(rng, 2, 200_000)
    near = rng.random(len(a)) < 0.3  # products beside 2^-126
    a = np.where(near, np.ldexp(F(1.0) + rng.integers(-40, 40, len(a)).astype(F) * F(2.0 ** -24), -60), a).astype(F)
    b = np.where(near, np.ldexp(F(1.0) + rng.integers(-40, 40, len(a)).astype(F) * F(2.0 ** -24), -66), b).astype(F)
    keep = np.isfinite(a) & np.isfinite(b) & (a > 0) & (b > 0)
    a, b = np.ascontiguousarray(a[keep]), np.ascontiguousarray(b[keep])
    out, split = np.zeros(len(a), F), np.zeros(len(a), F)
    rules.rule_product2(pointer(a), pointer(b), C.c_uint64(len(a)), pointer(out), pointer(split))
    assert same_bits(out, split)


@pytest.mark.parametrize("heuristic", [0, 1])
def test_mis_weights_equal_those_of_the_split_ratio(rules, heuristic):
    rng = np.random.default_rng(11 + heuristic)
    a, b = factors(rng, 2, 200_000)
    keep = np.isfinite(a) & np.isfinite(b) & (a > 0) & (b > 0)
    a, b = np.ascontiguousarray(a[keep]), np.ascontiguousarray(b[keep])
    weight, ratio = np.zeros(len(a), F), np.zeros(len(a), F)
    rules.rule_mis_weight(heuristic, pointer(a), pointer(b), C.c_uint64(len(a)), pointer(weight))
    less, more = np.minimum(a, b), np.maximum(a, b)
    rules.rule_split_mis_ratio(heuristic, pointer(less), pointer(more), C.c_uint64(len(a)), pointer(ratio))
    wanted = np.where(a < b, np.where(ratio > 0, ratio / (F(1.0) + ratio), F(1.0)), F(1.0) / (F(1.0) + ratio)).astype(F)
    assert same_bits(weight, wanted)


def test_next_float_is_nextafter(rules):
    rng = np.random.default_rng(13)
    v = rng.integers(0, 1 << 32, 300_000, dtype=np.uint32).view(F)
    v = np.concatenate([v[~np.isnan(v)], np.array([0.0, -0.0, MIN_NORMAL, -MIN_NORMAL, MAX_FLOAT, -MAX_FLOAT, 1e-45,
                                                   -1e-45, np.inf, -np.inf], F)])
    for up in (0, 1):
        out = np.zeros(len(v), F)
        rules.rule_next_float(pointer(v), up, C.c_uint64(len(v)), pointer(out))
        with np.errstate(all="ignore"):
            assert same_bits(out, np.nextafter(v, F(np.inf) if up else F(-np.inf)))


def triangles_and_rays(size, distance, n, seed):
    """Triangles of a size seen from a distance, half of the rays aimed near an edge."""
    rng = np.random.default_rng(seed)
    v = (rng.normal(size=(n, 3, 3)) * size).astype(F)
    w = rng.dirichlet((1.0, 1.0, 1.0), n)
    w[::2, 0] = rng.normal(size=len(w[::2])) * 10.0 ** rng.uniform(-9.0, 0.0, len(w[::2]))
    target = (w[:, :, None] * v).sum(axis=1) / w.sum(axis=1, keepdims=True)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(F)
    return v, (target - distance * d).astype(F), d


def run_triangles(rules, v, o, d):
    n = len(v)
    certain, code, out = np.zeros(n, np.uint8), np.zeros(n, np.uint8), np.zeros((n, 4), F)
    rules.rule_triangles(pointer(np.ascontiguousarray(v)), pointer(o), pointer(d), C.c_uint64(n), pointer(certain),
                         pointer(code), pointer(out))
    return certain != 0, code, out


@pytest.mark.parametrize("distance", [1e-3, 1.0, 30.0, 1e4, 1e12, 1e20])
@pytest.mark.parametrize("size", [1e-12, 1e-3, 1.0, 1e18, 1e20])
def test_certain_misses_are_misses(rules, size, distance):
    v, o, d = triangles_and_rays(size, distance, 3000, abs(int(np.log10(size) * 31 + np.log10(distance))))
    certain, code, _ = run_triangles(rules, v, o, d)
    assert (code[certain] == 0).all()
    for k in np.nonzero(certain)[0]:
        signs = exact_signs(list(v[k]), o[k], d[k])
        assert 1 in signs and -1 in signs, k
    if size / distance >= 1e-3 and 1e-10 < size < 1e10:  # near enough for the rule to decide anything
        assert certain.any()


def test_non_finite_rays_are_no_certain_misses(rules):
    v, o, d = triangles_and_rays(1.0, 1.0, 600, 3)
    for k, value in enumerate((np.nan, np.inf, -np.inf)):
        o[k::6, k] = value
        d[3 + k::6, k] = value
    certain, _, _ = run_triangles(rules, v, o, d)
    assert not certain.any()


def nearest_float(q):
    """The float32 nearest to a Fraction, ties to even."""
    f = F(float(q))
    best = min((F(np.nextafter(f, F(-np.inf))), f, F(np.nextafter(f, F(np.inf)))),
               key=lambda c: (abs(Fraction(float(c)) - q), int(c.view(np.uint32)) & 1))
    return best


@pytest.mark.parametrize("distance", [1.0, 100.0, 1e4])
@pytest.mark.parametrize("size", [1e-12, 1.0, 1e12])
def test_hits_are_the_exact_quotients_rounded_once(rules, size, distance):
    v, o, d = triangles_and_rays(size, distance * size, 400, int(distance) + 5)
    _, code, out = run_triangles(rules, v, o, d)
    assert (code != 2).all() and (code == 1).mean() > 0.3
    for k in range(len(v)):
        p = [[Fraction(float(v[k][j][a])) - Fraction(float(o[k][a])) for a in range(3)] for j in range(3)]
        r = [Fraction(float(x)) for x in d[k]]

        def det(a, b, c):
            return (a[0] * (b[1] * c[2] - b[2] * c[1]) - a[1] * (b[0] * c[2] - b[2] * c[0])
                    + a[2] * (b[0] * c[1] - b[1] * c[0]))

        e = [det(p[1], p[2], r), det(p[2], p[0], r), det(p[0], p[1], r)]
        total = sum(e)
        inside = total != 0 and (all(x >= 0 for x in e) or all(x <= 0 for x in e))
        t = det(p[0], p[1], p[2]) / total if inside else None
        assert (code[k] == 1) == (inside and t >= 0), k
        if code[k] == 1:
            wanted = [nearest_float(t)] + [nearest_float(x / total) for x in e]
            assert same_bits(out[k] + F(0.0), np.array(wanted, F) + F(0.0)), k  # a zero's sign is not compared
