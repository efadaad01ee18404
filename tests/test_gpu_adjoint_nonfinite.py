"""Infinities in a differentiable render reach the gradient as the reverse
sweep's products give them, also behind a cell so thick that nothing of the
adjoint passes it (0 times infinity is not 0): the sweep of the record against
the rays traced again."""

import numpy as np
import pytest

from grt import workloads

pytestmark = pytest.mark.gpu


def test_the_recorded_sweep_keeps_what_is_not_finite(gpu):
    w = workloads.scaled(workloads.C4, pixels=33, grid=(32, 16, 16), image_nx=33, image_ny=33)
    p, grid = w.params(), w.torus()
    shape = grid["r.npy"].shape
    rng = np.random.default_rng(3)
    m_abs = np.where(rng.random(shape) < 0.1, 1e15, 1.0)    # a tenth of the cells lets nothing through,
    m_emis = np.where(rng.random(shape) < 0.05, np.inf, 1.0)  # a twentieth shines without bound
    weights = np.random.default_rng(2).normal(size=(33, 33))
    out = []
    for again in (False, True):
        with gpu.Context(p) as ctx:
            ctx.upload_grid(grid)
            ctx.set_cell_multipliers(m_abs, m_emis)
            ctx.init_image_forward_photons(33, 33, workloads.C4_BACK_DISTANCE)
            ctx.forward_checkpointed(64)
            if again:
                ctx.set_params(p)  # every ray is traced again
            out.append(ctx.adjoint_image_I(weights, shape))
    for got, want in zip(*out):
        assert np.array_equal(np.isfinite(got), np.isfinite(want))
        here = np.isfinite(want)
        assert np.abs(got[here] - want[here]).max() <= 1e-12 * np.abs(want[here]).max()
    assert not np.isfinite(out[1][0]).all() and np.isfinite(out[1][0]).any()
