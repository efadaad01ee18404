"""The FP32 cell lookups at positions so close to the polar axis that the
arguments of the azimuth leave the range of FP32: the reference's cell, or left
to it."""

import ctypes as C

import numpy as np
import pytest

from test_gpu_division import LIB, dp

pytestmark = pytest.mark.gpu
_IP = C.POINTER(C.c_int)


@pytest.mark.parametrize("scale", [1.0, 1e-10, 1e10])
@pytest.mark.parametrize("spin", [0.0, 0.94])
@pytest.mark.parametrize("bend", [0.0, 0.05])
def test_positions_near_the_axis(gpu, scale, spin, bend):
    selftest = C.CDLL(str(LIB))
    rng = np.random.default_rng(4)
    n = 200_000
    r = np.ascontiguousarray(scale * np.exp(np.linspace(np.log(1.3), np.log(50.0), 40)))
    th = np.linspace(0.01, np.pi - 0.01, 24)  # the axis lies inside the first and the last cell
    k = np.arange(20)
    ph = np.ascontiguousarray(2 * np.pi * (k + bend * np.sin(k)) / 20)
    off = scale * 10.0 ** rng.uniform(-320, 0, n)  # from the axis; the smallest are zeros and subnormals
    az = rng.uniform(0, 2 * np.pi, n)
    pos = np.ascontiguousarray(np.column_stack([off * np.cos(az), off * np.sin(az),
                                                scale * rng.uniform(1.3, 50.0, n) * rng.choice([-1.0, 1.0], n)]))
    even, stretched, exact = (np.empty(n, dtype=np.int32) for _ in range(3))
    is_even = C.c_int(-1)
    assert selftest.grt_selftest_locate(dp(r), r.size, dp(th), th.size, dp(ph), ph.size, C.c_double(spin * scale), dp(pos),
                                        C.c_size_t(n), *(v.ctypes.data_as(_IP) for v in (even, stretched, exact)),
                                        C.byref(is_even)) == 0
    assert is_even.value == int(bend == 0.0)
    for fast in (even, stretched):
        decided = fast != -2
        assert np.array_equal(fast[decided], exact[decided])
    if is_even.value:
        assert (even != -2)[off > 1e-12 * scale].mean() > 0.9
