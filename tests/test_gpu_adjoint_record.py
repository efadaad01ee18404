"""The adjoint sweeps the transfer updates that the checkpointed forward
recorded; rays with more updates than a ray's share of the record, and every ray
once the parameters or the grid changed, are traced again from their
checkpoints.  All three give the same gradient."""

import math

import numpy as np
import pytest

from grt import workloads

pytestmark = pytest.mark.gpu


def gradient(gpu, w, weights, K, touch=None, **kw):
    p, grid = w.params(), w.torus()
    p.update(**kw)
    rng = np.random.default_rng(8)
    shape = grid["r.npy"].shape
    with gpu.Context(p) as ctx:
        ctx.upload_grid(grid)
        ctx.set_cell_multipliers(np.exp(rng.normal(0, 0.1, shape)), np.exp(rng.normal(0, 0.1, shape)))
        ctx.init_image_forward_photons(w.pixels, w.pixels, workloads.C4_BACK_DISTANCE)
        ctx.forward_checkpointed(K)
        steps = ctx.image_products().image_I
        if touch == "params":
            ctx.set_params(p)
        elif touch == "grid":
            ctx.upload_grid(grid)
        ga, ge = ctx.adjoint_image_I(weights, shape)
        return steps, ga, ge


@pytest.mark.parametrize("pixels", [7, 33])
@pytest.mark.parametrize("K", [3, 64])
def test_recorded_and_recomputed_sweeps_agree(gpu, pixels, K):
    w = workloads.scaled(workloads.C4, pixels=pixels, grid=(32, 16, 16), image_nx=pixels, image_ny=pixels)
    weights = np.random.default_rng(9).normal(size=(pixels, pixels))
    image, ga, ge = gradient(gpu, w, weights, K)
    assert np.abs(ga).max() > 0 and np.abs(ge).max() > 0
    for touch in ("params", "grid"):
        again, ga2, ge2 = gradient(gpu, w, weights, K, touch)
        # sums of the same terms in the order of their atomic additions: at most
        # a few hundred per pixel or cell, each rounding at 2^-53 of the partial sum
        for a, b in ((image, again), (ga, ga2), (ge, ge2)):
            assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


def test_rays_beyond_their_share_of_the_record(gpu):
    # small fixed steps inside the torus: several hundred sampled steps a ray
    w = workloads.scaled(workloads.C4, pixels=9, grid=(32, 16, 16), image_nx=9, image_ny=9)
    kw = dict(integrator=0, initial_step=0.2 / workloads.C4_BACK_DISTANCE, max_steps=2000)
    weights = np.random.default_rng(10).normal(size=(9, 9))
    _, ga, ge = gradient(gpu, w, weights, 64, **kw)
    _, ga2, ge2 = gradient(gpu, w, weights, 64, "params", **kw)
    assert np.abs(ge).max() > 0 and math.isfinite(np.abs(ga).max())
    for a, b in ((ga, ga2), (ge, ge2)):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
