"""Rays at random screen positions are queued by screen cell.  The order is a
permutation that changes no ray: against the same photons uploaded to a context
without images, which traces them in the order they were drawn -- sizes around
the steps of the cell grid, a window far from square, and photons put back into
the initialised slots."""

import numpy as np
import pytest

from grt import abi
from grt import workloads
from helpers import mini

pytestmark = pytest.mark.gpu


def fields(ph):
    return [getattr(ph, f).view(np.uint8) for f in abi.PHOTON_FIELDS]


@pytest.mark.parametrize("n", [1, 7, 8, 9, 32, 33, 129, 4097, 90001])
@pytest.mark.parametrize("height", [40.0, 0.5])
def test_screen_order_changes_no_ray(gpu, n, height):
    w = mini(workloads.C2, 16, (24, 16, 16), camera_height=height)
    p, grid = w.params(), w.torus()
    with gpu.Context(p) as ctx:
        ctx.upload_grid(grid)
        ctx.init_image_photons_random(n)
        start = ctx.download_photons()
        stats = ctx.run()
        got = ctx.download_photons()
        ctx.upload_photons(start)  # the same slots
        ctx.run()
        again = ctx.download_photons()
    with gpu.Context(p) as ctx:
        ctx.upload_grid(grid)
        ctx.upload_photons(start)
        wstats = ctx.run()
        want = ctx.download_photons()
    assert stats["accepted_steps"] == wstats["accepted_steps"] and stats["n_terminated"] == n
    for a, b, c in zip(fields(got), fields(want), fields(again)):
        assert np.array_equal(a, b) and np.array_equal(a, c)
