"""The shading header's own product, MIS and stepping rules, compiled for the host (tests/device_rules.cpp):
float32 operations round there as on the device, so what holds here holds in the kernels."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

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
