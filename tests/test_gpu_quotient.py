"""The samplers' packed quotient equals the IEEE division bit for bit on the operands it is used for: numerators of at
least 2^-30, quotients of 2^-100 to 2^29. Its last step rounds correctly when the reciprocal before it is the correctly
rounded one, which that theorem leaves open for one divisor significand, all ones; here that one is checked against
every numerator, and every divisor against hard numerators."""
import ctypes

import numpy as np
import pytest

from csdecomp_b200 import _capi

pytestmark = pytest.mark.gpu

ALL = (np.arange(1 << 23, dtype=np.uint32) | np.uint32(0x3F800000)).view(np.float32)  # every significand, [1, 2)
ONES = np.array([0x3FFFFFFF], np.uint32).view(np.float32)


def mismatches(s, a, paired=False):
    s, a = np.ascontiguousarray(s, np.float32), np.ascontiguousarray(a, np.float32)
    n, ex = ctypes.c_int64(-1), np.zeros(2, np.float32)
    _capi.check(_capi.lib().csd_quotient_probe(_capi.ptr(s), ctypes.c_int64(s.size), _capi.ptr(a), ctypes.c_int64(a.size),
                                               int(paired), ctypes.byref(n), _capi.ptr(ex)))
    return n.value, [float(x).hex() for x in ex]


def significands(rng, n):
    return rng.integers(0, 1 << 23, n, dtype=np.uint32)


def test_the_all_ones_divisor_against_every_numerator():
    for scale in (1.0, -1.0, 2.0 ** -20, 2.0 ** 100):
        n, ex = mismatches(ALL, ONES * np.float32(scale))
        assert n == 0, ex


def test_every_divisor_against_boundary_numerators():
    edge = np.array([0, 1, 2, 3, 0x3FFFFF, 0x400000, 0x400001, 0x2AAAAA, 0x555555, 0x7FFFFC, 0x7FFFFD, 0x7FFFFE, 0x7FFFFF],
                    np.uint32)
    n, ex = mismatches((edge | np.uint32(0x3F800000)).view(np.float32), ALL)
    assert n == 0, ex


def test_boundary_and_random_divisors_against_every_numerator():
    rng = np.random.default_rng(1)
    edge = np.array([0, 1, 2, 0x3FFFFF, 0x400000, 0x555555, 0x2AAAAA, 0x7FFFFC, 0x7FFFFD, 0x7FFFFE], np.uint32)
    m = np.concatenate([edge, significands(rng, 500)])
    n, ex = mismatches(ALL, (m | np.uint32(0x3F800000)).view(np.float32))
    assert n == 0, ex


@pytest.mark.parametrize("seed", range(8))
def test_quotients_nearest_a_rounding_midpoint(seed):
    """Numerators next to a (q + half an ulp), where a quotient off by less than its last bit's half rounds wrongly."""
    rng = np.random.default_rng(seed)
    k = 1 << 22
    a = (significands(rng, k) | np.uint32(0x3F800000)).view(np.float32).astype(np.float64)
    if seed % 2:
        a = np.float64(2) - np.ldexp(rng.integers(1, 1 << 10, k).astype(np.float64), -23)  # near the all-ones divisor
    q = (significands(rng, k) | np.uint32(0x3F800000)).view(np.float32).astype(np.float64) + 2.0 ** -24
    s = (a * q).astype(np.float32)  # the nearest numerator
    for d in (s, np.nextafter(s, np.float32(0)), np.nextafter(s, np.float32(np.inf))):
        n, ex = mismatches(d, a.astype(np.float32), paired=True)
        assert n == 0, ex


@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_both_ends_of_the_range(sign):
    """Numerators from 2^-30 to the largest, divisors so that the quotient spans [2^-100, 2^29)."""
    rng = np.random.default_rng(3)
    k = 1 << 23
    es = rng.integers(-30, 128, k)
    es[: k // 4] = -30
    es[k // 4: k // 2] = 127
    eq = rng.integers(-100, 29, k)
    eq[::3] = -100
    eq[1::3] = 28
    s = np.ldexp(1.0 + significands(rng, k) / 2.0 ** 23, es)
    q = np.ldexp(1.0 + significands(rng, k) / 2.0 ** 23, eq)
    a = s / q
    ok = (np.abs(a) < 2.0 ** 126) & (np.abs(a) >= 2.0 ** -126)
    s, a = s[ok].astype(np.float32), (sign * a[ok]).astype(np.float32)
    quo = np.abs(s.astype(np.float64) / a)
    ok = (quo >= 2.0 ** -100) & (quo < 2.0 ** 29) & (np.abs(a) < 2.0 ** 126)
    assert ok.sum() > k // 2
    n, ex = mismatches(s[ok], a[ok], paired=True)
    assert n == 0, ex
