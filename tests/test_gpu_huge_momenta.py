"""Momenta close to overflow (rays that hang at the horizon when termination.r_min
lies inside it reach them) and to underflow: the kernels' right-hand side, with
its factors of two moved, and the RK4 step overflow exactly where the
reference's expressions do.

* ks_rhs_rcp against ks_rhs, bit for bit wherever it does not hand the state on,
  and it keeps every state with momenta of an ordinary size;
* RK45 runs of photons with such momenta against the oracle, every field
  bit for bit, infinities included, NaN for NaN."""

import numpy as np
import pytest

from grt import abi, workloads
from helpers import run_gpu, run_oracle
from test_gpu_division import assert_bitwise, random_states, rhs, selftest  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spin", [0.0, 0.94])
def test_right_hand_side_at_any_momentum(selftest, spin):  # noqa: F811
    rng = np.random.default_rng(21)
    n = 1 << 19
    s = random_states(rng, n, spin)
    e = rng.integers(-1070, 1024, n)
    e[: n // 2] = rng.integers(500, 513, n // 2)  # the squares of these overflow, or just do not
    s[:, 3:] *= 0.9
    s[:, 3:] = np.ldexp(s[:, 3:], e[:, None])
    with np.errstate(all="ignore"):
        fast, ieee, inside = rhs(selftest, s, spin)
    assert_bitwise(fast.ravel(), ieee.ravel(), np.repeat(inside, 7))
    assert inside[np.abs(e) < 250].mean() > 0.99


def photons(gpu, p, rng, pixels, spin, radii, sizes, steps):
    """pixels^2 photons at random places with momenta of the given sizes and steps that change them by their own size."""
    n = pixels * pixels
    with gpu.Context(p) as ctx:
        ctx.upload_grid(None)
        ctx.init_image_photons(pixels, pixels)
        ph = ctx.download_photons()
    s = random_states(rng, n, spin)
    r = np.sqrt((s[:, :3] ** 2).sum(axis=1))
    s[:, :3] *= (rng.uniform(*radii, n) / r)[:, None]
    size = 10.0 ** sizes
    for f, v in zip(("x1", "x2", "x3"), s[:, :3].T):
        getattr(ph, f)[:] = v
    for f, v in zip(("k0", "k1", "k2", "k3"), s[:, 3:].T):
        getattr(ph, f)[:] = 0.5 * v * size
    ph.dlambda[:] = rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(*steps, n) / size
    return ph


def assert_same_bits(got, want):
    n = got.n
    for f in abi.PHOTON_FIELDS:
        a, b = getattr(got, f), getattr(want, f)
        same = (a.view(np.uint8).reshape(n, -1) == b.view(np.uint8).reshape(n, -1)).all(axis=1)
        same |= np.isnan(a.astype(np.float64)) & np.isnan(b.astype(np.float64))
        assert same.all(), (f, (~same).sum(), np.flatnonzero(~same)[:5], a[~same][:3], b[~same][:3])


@pytest.mark.parametrize("spin", [0.0, 0.94])
def test_rk45_with_huge_momenta_is_the_oracles(gpu, oracle, spin):
    rng = np.random.default_rng(22)
    w = workloads.ImageWorkload("huge", (16, 8, 8), spin, 60.0, 100, abi.RK45, 0.01, 3)
    p, grid, n = w.params().update(camera_distance=100.0, r_term_max=150.0, r_term_min=0.5), w.torus(), 10000
    sizes = np.where(rng.random(n) < 0.7, rng.uniform(152.0, 155.5, n), rng.uniform(100.0, 308.0, n))
    ph = photons(gpu, p, rng, 100, spin, (2.2, 60.0), sizes, (-3, 1))
    got, _, gst = run_gpu(gpu, p, grid, photons=ph)
    want, _, wst = run_oracle(oracle, p, grid, photons=ph)
    assert_same_bits(got, want)
    assert gst["accepted_steps"] == wst["accepted_steps"] and (want.terminate == 1).any()


@pytest.mark.parametrize("spin", [0.0, 0.94])
def test_an_rk4_step_overflows_as_the_oracles(gpu, oracle, spin):
    """2 k2 and 2 k3 overflow by themselves, whatever the sum they go into."""
    rng = np.random.default_rng(1)
    w = workloads.ImageWorkload("huge", (16, 8, 8), spin, 60.0, 300, abi.RK4, 0.01, 1)
    p, grid = w.params().update(camera_distance=100.0, r_term_max=1e6, r_term_min=0.5), w.torus()
    ph = photons(gpu, p, rng, 300, spin, (2.2, 10.0), rng.uniform(153.5, 154.8, 90000), (0, 1.5))
    got, _, _ = run_gpu(gpu, p, grid, photons=ph)
    want, _, _ = run_oracle(oracle, p, grid, photons=ph)
    assert_same_bits(got, want)
    assert np.isnan(want.k1).any() and np.isfinite(want.k1).any()
