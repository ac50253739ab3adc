"""The mathematics of the rule by which shading multiplies factors directly instead of by frexp significands
(Factors::direct in bf200_shading.cuh): whenever it applies, both forms have the same bits. Restated
here in numpy float32, whose operations round like the device's; test_device_rules.py checks the
header's own code."""
import numpy as np
import pytest

F = np.float32
MIN_NORMAL, MAX_FLOAT = F(1.17549435e-38), F(3.40282347e+38)


def direct(num, den):
    product, least = num[0].copy(), num[0].copy()
    for v in num[1:]:
        product = product * v
        least = np.fmin(least, np.fmin(v, product))
    for v in den:
        product = product / v
        least = np.fmin(least, np.fmin(v, product))
    return product, (least > MIN_NORMAL) & (product <= MAX_FLOAT)


def split(num, den, renormalise):
    """The exponent-split form: checked_product_quotient, or checked_product_ratio (renormalise)."""
    significand, exponent = np.ones_like(num[0]), np.zeros(num[0].shape, np.int64)
    for values, sign in ((num, 1), (den, -1)):
        for v in values:
            m, e = np.frexp(v)
            significand = significand * m if sign > 0 else significand / m
            exponent = exponent + sign * e
            if renormalise:
                significand, n = np.frexp(significand)
                exponent = exponent + n
    significand, n = np.frexp(significand)
    return np.ldexp(significand, np.clip(exponent + n, -400, 400).astype(np.int32))


def factors(rng, count, n):
    """Factors over the whole float range: moderate, extreme, powers of two, subnormal, zero, negative,
    infinite and NaN ones."""
    out = []
    for _ in range(count):
        spread = rng.choice([1.0, 8.0, 40.0, 126.0], n)
        v = (np.exp2(rng.uniform(-1.0, 1.0, n) * spread)).astype(F)
        odd = rng.random(n)
        v = np.where(odd < 0.02, F(0.0), v)
        v = np.where((odd >= 0.02) & (odd < 0.04), np.exp2(np.round(np.log2(np.maximum(v, MIN_NORMAL)))), v)
        v = np.where((odd >= 0.04) & (odd < 0.06), F(1e-40), v)
        v = np.where((odd >= 0.06) & (odd < 0.07), -v, v)
        v = np.where((odd >= 0.07) & (odd < 0.08), F(np.inf), v)
        v = np.where((odd >= 0.08) & (odd < 0.09), F(np.nan), v)
        v = np.where((odd >= 0.09) & (odd < 0.1), MAX_FLOAT, v)
        out.append(v.astype(F))
    return out


@pytest.mark.parametrize("renormalise", [False, True])
@pytest.mark.parametrize("counts", [(2, 1), (3, 1), (4, 1), (2, 2), (5, 2), (7, 2), (7, 4)])
def test_direct_products_equal_the_split_form(counts, renormalise):
    rng = np.random.default_rng(17 * counts[0] + counts[1])
    num, den = factors(rng, counts[0], 200_000), factors(rng, counts[1], 200_000)
    with np.errstate(all="ignore"):
        product, applies = direct(num, den)
        expected = split(num, den, renormalise)
    assert 0.05 < applies.mean() < 1.0
    assert np.array_equal(product[applies].view(np.uint32), expected[applies].view(np.uint32))
    valid = np.all([np.isfinite(v) & (v > 0) for v in num + den], axis=0)
    assert valid[applies].all()


def test_direct_mis_ratios_equal_the_split_form():
    rng = np.random.default_rng(3)
    a, b = factors(rng, 2, 400_000)
    keep = np.isfinite(a) & np.isfinite(b) & (a > 0) & (b > 0)
    n, d = np.minimum(a[keep], b[keep]), np.maximum(a[keep], b[keep])
    with np.errstate(all="ignore"):
        plain = n / d
        ms, me = np.frexp(n)
        ds, de = np.frexp(d)
        r = ms / ds
        for power in (1, 2):
            ratio = plain if power == 1 else plain * plain
            applies = np.fmin(np.fmin(n, plain), ratio) >= MIN_NORMAL
            exponent = np.clip(power * (me - de), -400, 400).astype(np.int32)
            expected = np.ldexp(r if power == 1 else r * r, exponent)
            assert 0.05 < applies.mean() < 1.0
            assert np.array_equal(ratio[applies].view(np.uint32), expected[applies].view(np.uint32))


def test_next_float_steps():
    """next_float: one step of the bit pattern is nextafter for every finite value."""
    rng = np.random.default_rng(5)
    bits = rng.integers(0, 1 << 32, 500_000, dtype=np.uint32)
    v = np.concatenate([bits.view(F), np.array([0.0, -0.0, MIN_NORMAL, -MIN_NORMAL, MAX_FLOAT, -MAX_FLOAT, 1e-45], F)])
    v = v[np.isfinite(v)]
    for up in (True, False):
        step = np.where((v > 0) == up, 1, -1).astype(np.int32)
        stepped = (v.view(np.int32) + step).view(F)
        stepped = np.where(v == 0, F(1e-45) if up else F(-1e-45), stepped)
        with np.errstate(all="ignore"):
            expected = np.nextafter(v, F(np.inf) if up else F(-np.inf))
        assert np.array_equal(stepped.view(np.uint32), expected.view(np.uint32))


def test_unit_normals_by_one_reciprocal_root():
    """transform_normal's rule: where the float around a reciprocal-root normal is certain (2^-46), the
    divided and scaled form rounds to it too."""
    rng = np.random.default_rng(9)
    v = rng.normal(size=(400_000, 3)) * np.exp2(rng.uniform(-60.0, 60.0, (400_000, 1)))
    v[::5, 0] *= np.exp2(rng.uniform(-40.0, 0.0, len(v[::5])))
    v[::7, 1] = 0.0
    squared = v[:, 0] * v[:, 0] + (v[:, 1] * v[:, 1] + v[:, 2] * v[:, 2])
    root = 1.0 / np.sqrt(squared)
    root = root * (1.0 + rng.choice([-2.0, 0.0, 2.0], len(v)) * 2.0 ** -52)  # a root some ulps off
    q = v * root[:, None]
    slack = np.abs(q) * 2.0 ** -46
    low, high = (q - slack).astype(F), (q + slack).astype(F)
    certain = (low == high).all(axis=1)
    scaled = v / np.abs(v).max(axis=1, keepdims=True)
    length = np.sqrt(scaled[:, 0] * scaled[:, 0] + (scaled[:, 1] * scaled[:, 1] + scaled[:, 2] * scaled[:, 2]))
    expected = (scaled / length[:, None]).astype(F)
    assert certain.mean() > 0.999
    assert np.array_equal(low[certain].view(np.uint32), expected[certain].view(np.uint32))
