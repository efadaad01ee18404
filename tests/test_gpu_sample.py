"""The fluid sample's short cuts decide as the reference's arithmetic does.

* The FP32 cell lookups (locate_even on grids even in log r, theta, phi;
  locate_stretched on any separable grid) against locate_exact: the same cell
  or the same rejection wherever they decide, on positions over the whole grid
  and its surroundings, next to cell edges and next to the polar axis; and they
  decide nearly always.
* tetrad_certain against build_tetrad: never true where there is no tetrad.
* Scattering packets that wait for company: a run cut into launches of three
  calls, and one stopped by its iteration limit, leave every packet at the state
  that calls taken one by one give."""

import ctypes as C

import numpy as np
import pytest

from grt import abi, torus, workloads
from test_gpu_division import LIB, dp

pytestmark = pytest.mark.gpu
_IP = C.POINTER(C.c_int)


@pytest.fixture(scope="module")
def selftest(gpu):
    return C.CDLL(str(LIB))


def axes(kind, nr, nth, nph):
    r = np.exp(np.linspace(np.log(1.3), np.log(50.0), nr)) if nr > 1 else np.array([5.0])
    th = np.linspace(0.01, np.pi - 0.01, nth) if nth > 1 else np.array([1.5])
    ph = np.linspace(0.0, 2 * np.pi, nph, endpoint=False)
    if kind == "shifted":
        th = (np.arange(nth) + 0.5) * np.pi / nth
        ph = ph + np.pi / nph
    elif kind == "stretched":
        r = 1.3 + (r - 1.3) ** 1.5
        th = np.pi * (0.5 + 0.5 * np.sin(np.linspace(-1.5, 1.5, nth)) / np.sin(1.5)) * 0.98 + 0.03
    elif kind == "wedge":
        ph = np.linspace(0.3, 1.4, nph)
    return r, th, ph


def positions(rng, n, r, th, ph, spin):
    """Random positions, and positions at and next to the midpoints and the ends of the cells."""
    q = [np.exp(rng.uniform(np.log(r[0] * 0.8), np.log(r[-1] * 1.2), n)), np.arccos(rng.uniform(-1, 1, n)),
         rng.uniform(0, 2 * np.pi, n)]
    for k, axis in enumerate((np.log(r), th, ph)):
        if axis.size < 2:
            continue
        i = rng.integers(-1, axis.size, n // 4)
        gap = np.diff(axis)
        edge = np.where(i < 0, axis[0] - gap[0] / 2, np.where(i >= axis.size - 1, axis[-1] + gap[-1] / 2,
                        (axis[np.clip(i, 0, axis.size - 2)] + axis[np.clip(i, 0, axis.size - 2) + 1]) / 2))
        edge = edge + rng.choice([0.0, 1e-15, -1e-12, 1e-9, 1e-7, -1e-6, 3e-6, -3e-5, 1e-4], n // 4) * gap[0]
        where = rng.permutation(n)[: n // 4]
        q[k][where] = np.exp(edge) if k == 0 else edge
    q[1][: n // 50] = rng.choice([0.0, 1e-12, 1e-7, 1e-4, np.pi - 1e-6], n // 50)
    R, T, P = q
    return np.ascontiguousarray(np.column_stack([(R * np.cos(P) - spin * np.sin(P)) * np.sin(T),
                                                 (R * np.sin(P) + spin * np.cos(P)) * np.sin(T), R * np.cos(T)]))


@pytest.mark.parametrize("kind", ["even", "shifted", "stretched", "wedge"])
@pytest.mark.parametrize("size", [(128, 64, 64), (97, 49, 35), (3, 2, 4), (40, 301, 7), (1, 1, 3), (700, 16, 500)])
def test_fp32_lookups_give_the_reference_cell(selftest, kind, size):
    rng = np.random.default_rng(sum(size))
    n = 200_000
    for spin in (0.0, 0.94, -0.5):
        r, th, ph = (np.ascontiguousarray(a) for a in axes(kind, *size))
        pos = positions(rng, n, r, th, ph, spin)
        even, stretched, exact = (np.empty(n, dtype=np.int32) for _ in range(3))
        is_even = C.c_int(-1)
        rc = selftest.grt_selftest_locate(dp(r), r.size, dp(th), th.size, dp(ph), ph.size, C.c_double(spin), dp(pos),
                                          C.c_size_t(n), *(v.ctypes.data_as(_IP) for v in (even, stretched, exact)),
                                          C.byref(is_even))
        assert rc == 0
        assert is_even.value == int(kind in ("even", "shifted") and min(size) > 1)
        for fast in (even, stretched):
            decided = fast != -2
            assert np.array_equal(fast[decided], exact[decided]), (kind, size, spin)
        # (3/4)^3 of the positions, 0.42, were moved next to no edge
        if is_even.value and max(size) < 200:
            assert (even != -2).mean() > 0.4
        if min(size) > 1 and kind != "wedge":
            assert (stretched != -2).mean() > 0.4


@pytest.mark.parametrize("spin", [0.0, 0.94, 1.0])
def test_certain_tetrads_exist(selftest, spin):
    rng = np.random.default_rng(5)
    n = 400_000
    pos = positions(rng, n, *axes("even", 64, 32, 32), spin)
    u = np.empty((n, 4))
    u[:, 0] = rng.normal(0, 1, n) * 10.0 ** rng.uniform(-3, 11, n)
    beta = np.where(rng.random(n) < 0.5, rng.uniform(0, 1.2, n), 1.0 - 10.0 ** rng.uniform(-12, 0, n))
    d = rng.normal(size=(n, 3))
    u[:, 1:] = d / np.linalg.norm(d, axis=1)[:, None] * (beta * np.abs(u[:, 0]))[:, None]
    u[: n // 100] = 0.0
    u[n // 100: n // 50, 1] = np.nan
    u[n // 50: n // 40, 0] = np.inf
    out = np.empty(n, dtype=np.uint32)
    rc = selftest.grt_selftest_tetrad(dp(pos), dp(u), C.c_size_t(n), C.c_double(spin), C.c_double(1.0),
                                      out.ctypes.data_as(C.POINTER(C.c_uint32)))
    assert rc == 0
    certain, rolled, straight = out & 1, (out >> 1) & 1, (out >> 2) & 1
    assert np.array_equal(rolled, straight)
    assert not np.any((certain == 1) & (rolled == 0))
    assert 0.2 < certain.mean() < 0.8


def _disk(**kw):
    w = workloads.DiskWorkload("disk", (32, 16, 16), 0.9, 40.0)
    return w.params().update(**kw), torus.benchmark_torus(*w.grid, spin=w.spin)


def _run(gpu, p, grid, **shape):
    with gpu.Context(p) as ctx:
        if shape:
            ctx.set_launch_config(**shape)
        ctx.upload_grid(grid)
        ctx.init_disk_photons()
        try:
            ctx.run()
        except gpu.GrtError as e:
            assert e.status == abi.GRT_ETIMEOUT and shape
        return np.column_stack([getattr(ctx.download_photons(), f).astype(np.float64) for f in abi.PHOTON_FIELDS])


def test_waiting_scatterings_survive_launch_ends(gpu):
    p, grid = _disk()
    want = _run(gpu, p, grid)
    cut = _run(gpu, p.copy().update(output_interval=3, termination_percent=1.0 - 1e-12), grid)
    assert np.array_equal(want, cut)


@pytest.mark.parametrize("limit", [3, 7, 12])
def test_a_stopped_run_leaves_packets_at_call_boundaries(gpu, limit):
    p, grid = _disk()
    got = _run(gpu, p, grid, max_iterations=limit, blocks_per_sm=2, refill_threshold=4)
    left = np.ones(len(got), dtype=bool)
    for calls in range(limit + 1):
        if calls == 0:  # as emitted
            with gpu.Context(p) as ctx:
                ctx.upload_grid(grid)
                ctx.init_disk_photons()
                ph = ctx.download_photons()
                state = np.column_stack([getattr(ph, f).astype(np.float64) for f in abi.PHOTON_FIELDS])
        else:
            state = _run(gpu, p.copy().update(max_steps=calls), grid)
        left &= ~np.all(got == state, axis=1)
    assert not left.any(), left.sum()
