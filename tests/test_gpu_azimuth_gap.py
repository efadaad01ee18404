"""Grids that leave a gap in azimuth: the FP32 lookup gives the reference's cell or
rejection wherever it decides, and decides nearly everywhere -- positions in the
gap would otherwise be looked up twice.  Wedges of any width, two cells opposite
one another, a single one."""

import ctypes as C

import numpy as np
import pytest

from test_gpu_division import LIB, dp

pytestmark = pytest.mark.gpu
_IP = C.POINTER(C.c_int)


@pytest.mark.parametrize("first,last,nph", [(0.3, 1.4, 12), (0.0, 0.2, 31), (0.0, 5.9, 20), (3.0, 3.5, 3), (0.1, 6.1, 2),
                                            (1.0, 4.1, 2), (0.0, 2.9, 2), (0.0, 3.3, 3), (2.0, 2.0, 1)])
@pytest.mark.parametrize("spin", [0.0, 0.94])
def test_positions_in_and_around_a_wedge(gpu, first, last, nph, spin):
    selftest = C.CDLL(str(LIB))
    rng = np.random.default_rng(6)
    n = 200_000
    r = np.ascontiguousarray(np.exp(np.linspace(np.log(1.3), np.log(50.0), 40)))
    th, ph = np.linspace(0.01, np.pi - 0.01, 24), np.linspace(first, last, nph)
    R, T, P = np.exp(rng.uniform(np.log(1.2), np.log(55.0), n)), np.arccos(rng.uniform(-1, 1, n)), rng.uniform(0, 2 * np.pi, n)
    near = rng.choice(np.concatenate([ph, [first - (last - first) / max(nph - 1, 1) / 2, last + (last - first) / max(nph - 1, 1) / 2]]), n // 4)
    P[: n // 4] = near + rng.choice([0.0, 1e-12, -1e-9, 1e-6, -1e-5, 3e-5, -1e-3], n // 4)
    pos = np.ascontiguousarray(np.column_stack([(R * np.cos(P) - spin * np.sin(P)) * np.sin(T),
                                                (R * np.sin(P) + spin * np.cos(P)) * np.sin(T), R * np.cos(T)]))
    even, stretched, exact = (np.empty(n, dtype=np.int32) for _ in range(3))
    is_even = C.c_int(-1)
    assert selftest.grt_selftest_locate(dp(r), r.size, dp(th), th.size, dp(ph), ph.size, C.c_double(spin), dp(pos),
                                        C.c_size_t(n), *(v.ctypes.data_as(_IP) for v in (even, stretched, exact)),
                                        C.byref(is_even)) == 0
    assert is_even.value == 0
    decided = stretched != -2
    assert np.array_equal(stretched[decided], exact[decided])
    assert (exact >= 0).any() and (exact < 0).any()
    if last - first < 2.0:
        assert decided[n // 4:].mean() > 0.95
