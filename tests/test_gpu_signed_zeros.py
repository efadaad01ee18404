"""The right-hand side keeps the signs of zeros: ks_rhs and ks_rhs_rcp against
the reference's expressions (kerr_schild_core.hpp:161-192) in Python's own
doubles, bit for bit, on states with exactly zero coordinates and momenta of
either sign."""

import itertools
import math

import numpy as np
import pytest

from test_gpu_division import assert_bitwise, dp, selftest  # noqa: F401

pytestmark = pytest.mark.gpu


def rhs(x, y, z, pt, px, py, pz, a, M):
    rsq = x * x + y * y + z * z
    A = rsq - a * a
    S = math.sqrt(A * A + 4.0 * ((a * z) * (a * z)))
    r = math.sqrt(0.5 * (A + S))
    one = 1.0 + A / S
    dr = (x * one / (2.0 * r), y * one / (2.0 * r), (z * one + 2.0 * (a * a) * z / S) / (2.0 * r))
    B = r * r + a * a
    l1, l2, l3 = (r * x + a * y) / B, (r * y - a * x) / B, z / r
    r2 = r * r
    r3 = r2 * r
    D = r3 * r + (a * z) * (a * z)
    H = M * r3 / D
    ldp = ((-pt + l1 * px) + l2 * py) + l3 * pz
    out = [-pt - (-(2.0 * H)) * ldp, px - 2.0 * H * l1 * ldp, py - 2.0 * H * l2 * ldp, pz - 2.0 * H * l3 * ldp]
    for k, d in enumerate(dr):
        dB = 2.0 * r * d
        d1 = ((d * x + r if k == 0 else d * x + a if k == 1 else d * x) - l1 * dB) / B
        d2 = ((d * y - a if k == 0 else d * y + r if k == 1 else d * y) - l2 * dB) / B
        d3 = ((1.0 if k == 2 else 0.0) - l3 * d) / r
        dD = 4.0 * r3 * d + (2.0 * (a * a) * z) if k == 2 else 4.0 * r3 * d
        dH = M * (3.0 * r2 * d * D - r3 * dD) / (D * D)
        out.append(dH * (ldp * ldp) + 2.0 * H * ldp * ((d1 * px + d2 * py) + d3 * pz))
    return out


@pytest.mark.parametrize("spin", [0.0, 0.9, -0.9])
def test_zeros_keep_their_signs(selftest, spin):  # noqa: F811
    places = itertools.product((0.0, -0.0, 3.0, -3.0), repeat=3)
    momenta = list(itertools.product((0.0, -0.0, 1.0, -1.0), repeat=4))
    states = np.array([(*q, *p) for q in places if any(q) and math.hypot(*q) > 1.0 for p in momenta])
    want = np.array([rhs(*s, spin, 1.0) for s in states.tolist()])
    fast, ieee = np.empty_like(want), np.empty_like(want)
    inside = np.empty(len(states), dtype=np.uint32)
    assert selftest.grt_selftest_rhs(dp(states), len(states), spin, 1.0, dp(fast), dp(ieee),
                                     inside.ctypes.data_as(selftest.grt_selftest_rhs.argtypes[6])) == 0
    # all but denominators with a low word of ones: without spin r^2 = 18 rounds to one
    inside = np.repeat(inside.astype(bool), 7)
    assert inside.mean() > 0.5
    assert_bitwise(ieee.ravel(), want.ravel())
    assert_bitwise(fast.ravel(), want.ravel(), inside)
    assert np.signbit(want[want == 0.0]).any()
