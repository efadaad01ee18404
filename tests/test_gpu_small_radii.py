"""The FP32 cell lookups on grids that reach far inside the hole.  There the
Kerr-Schild radius loses digits as (a / r)^2, and with it the polar angle
acos(z / r) of the reference's lookup, by more than the margins of the FP32
lookups: they have to leave such positions to it.  With spin 0 there is no such
loss and they decide down to the smallest radii."""

import ctypes as C

import numpy as np
import pytest

from test_gpu_division import LIB, dp

pytestmark = pytest.mark.gpu
_IP = C.POINTER(C.c_int)


@pytest.fixture(scope="module")
def selftest(gpu):
    return C.CDLL(str(LIB))


@pytest.mark.parametrize("stretch", [0.0, 0.1])
@pytest.mark.parametrize("nth", [16, 64, 1000])
@pytest.mark.parametrize("spin", [0.0, 0.94, -0.5, 1.0])
def test_lookups_far_inside_give_the_reference_cell(selftest, spin, nth, stretch):
    rng = np.random.default_rng(nth)
    n = 400_000
    r = np.ascontiguousarray(np.exp(np.linspace(np.log(1e-8), np.log(2.0), 120)))
    u = (np.arange(nth) + 0.5) / nth
    th = np.ascontiguousarray(np.pi * (u - stretch * np.sin(2 * np.pi * u) / (2 * np.pi)))
    ph = np.linspace(0.0, 2 * np.pi, 24, endpoint=False)
    R, T, P = np.exp(rng.uniform(np.log(r[0]), np.log(r[-1]), n)), np.arccos(rng.uniform(-1, 1, n)), rng.uniform(0, 2 * np.pi, n)
    pos = np.ascontiguousarray(np.column_stack([(R * np.cos(P) - spin * np.sin(P)) * np.sin(T),
                                                (R * np.sin(P) + spin * np.cos(P)) * np.sin(T), R * np.cos(T)]))
    even, stretched, exact = (np.empty(n, dtype=np.int32) for _ in range(3))
    is_even = C.c_int(-1)
    assert selftest.grt_selftest_locate(dp(r), r.size, dp(th), th.size, dp(ph), ph.size, C.c_double(spin), dp(pos),
                                        C.c_size_t(n), *(v.ctypes.data_as(_IP) for v in (even, stretched, exact)),
                                        C.byref(is_even)) == 0
    assert is_even.value == int(stretch == 0.0)
    for fast in (even, stretched):
        decided = fast != -2
        assert np.array_equal(fast[decided], exact[decided])
    # outside 0.01 |a| they still decide nearly always
    share = ((even if is_even.value else stretched) != -2)[R > 0.011 * abs(spin)].mean()
    assert share > (0.9 if nth < 1000 else 0.5)
