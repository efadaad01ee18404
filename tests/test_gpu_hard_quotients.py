"""div_by (grt_div.cuh) takes one residual step from a correctly rounded
reciprocal; its header argues that this is the IEEE quotient for every pair of
operands.  The pairs that come closest to breaking it are checked here, on the
GPU, bit for bit against IEEE division (the device's and numpy's):

* quotients next to a rounding midpoint: for an odd denominator B the
  numerators A with A 2^k = M B -+ j, M an odd 54-bit integer (a midpoint of
  two doubles) and j = 1, 3, the nearest a quotient can come to one;
* both significands just below 2, where the reciprocal's and the product's
  rounding errors can add up to 1.5 ulp, and just above 1.
"""

import random

import numpy as np
import pytest

from test_gpu_division import assert_bitwise, divide, selftest  # noqa: F401

pytestmark = pytest.mark.gpu


def hard_pairs(rng, count):
    a, b = [], []
    while len(a) < count:
        B = rng.getrandbits(52) | (1 << 52) | 1
        if rng.random() < 0.4:  # significands near 2
            B = 2 ** 53 - 1 - 2 * rng.getrandbits(rng.choice([3, 10, 26]))
        for k in (53, 54):  # quotients in [1, 2) and (1/2, 1)
            for j in (1, -1, 3, -3):
                M = pow(B, -1, 2 ** k) * j % 2 ** k
                M += 2 ** 53 if M < 2 ** 53 else 0
                A = (M * B - j) >> k
                if A << k == M * B - j and 2 ** 52 <= A < 2 ** 53:
                    a.append(A)
                    b.append(B)
    return np.array(a, dtype=np.float64), np.array(b, dtype=np.float64)


@pytest.mark.parametrize("exponent", [-420, 0, 397])
def test_hardest_quotients_are_ieee(selftest, exponent):  # noqa: F811
    a, b = hard_pairs(random.Random(31 + exponent), 20000)
    a, b = np.ldexp(a, exponent), np.ldexp(b, -exponent // 2)
    for sign in (1.0, -1.0):
        q, w = divide(selftest, a, sign * b)
        assert_bitwise(q, w)
        assert_bitwise(q, a / (sign * b))


def test_significands_at_the_ends_of_the_binade(selftest):  # noqa: F811
    m = np.arange(1, 513, dtype=np.float64)
    low, high = 2.0 ** 52 + m, 2.0 ** 53 - m
    for x in (low, high):
        for y in (low, high):
            a, b = (v.ravel() for v in np.meshgrid(x, y))
            q, w = divide(selftest, a, b)
            assert_bitwise(q, w)
            assert_bitwise(q, a / b)
