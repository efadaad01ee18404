"""Disk mode on a grid that is not separable, where the lookup scans the
coordinate arrays: packets scatter without waiting for others, and a run cut
into launches of three calls leaves every packet as one launch does."""

import numpy as np
import pytest

from grt import abi, torus, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norm", [1.0, 40.0])
def test_scatterings_on_a_bent_grid_survive_launch_ends(gpu, norm):
    w = workloads.DiskWorkload("disk", (24, 16, 16), 0.9, norm)
    grid = torus.benchmark_torus(*w.grid, spin=w.spin)
    grid = dict(grid, **{"theta.npy": grid["theta.npy"] + 1e-4 * np.sin(grid["r.npy"])})
    runs = []
    for kw in ({}, dict(output_interval=3, termination_percent=1.0 - 1e-12)):
        with gpu.Context(w.params().update(max_steps=90, **kw)) as ctx:
            ctx.upload_grid(grid)
            ctx.init_disk_photons()
            start = ctx.download_photons()
            ctx.run()
            runs.append(ctx.download_photons())
    for f in abi.PHOTON_FIELDS:
        assert np.array_equal(getattr(runs[0], f).view(np.uint8), getattr(runs[1], f).view(np.uint8)), f
    assert np.mean(runs[0].k1 != start.k1) > 0.5
