"""The refill threshold the library picks while no launch shape is set (32 in
image mode, 4 in disk mode) changes no photon: against the thresholds at the
ends of the range, set by hand, with more rays than the resident lanes so that
warps do refill."""

import numpy as np
import pytest

from grt import abi, torus, workloads

pytestmark = pytest.mark.gpu


def photons(gpu, p, grid, start, **shape):
    with gpu.Context(p) as ctx:
        if shape:
            ctx.set_launch_config(**shape)
        ctx.upload_grid(grid)
        start(ctx)
        stats = ctx.run()
        return ctx.download_photons().as_dict(), stats


@pytest.mark.parametrize("mode", ["image", "disk"])
def test_default_refill_gives_the_same_photons(gpu, mode):
    if mode == "image":
        w = workloads.scaled(workloads.C2, pixels=293, grid=(32, 16, 16), image_nx=293, image_ny=293)
        p, grid = w.params(), w.torus()
        start = lambda ctx: ctx.init_image_photons(293, 293)  # noqa: E731
    else:
        w = workloads.DiskWorkload("disk", (48, 24, 24), 0.9, 60.0)
        p, grid = w.params(), torus.benchmark_torus(*w.grid, spin=w.spin)
        start = lambda ctx: ctx.init_disk_photons()  # noqa: E731
    got, st = photons(gpu, p, grid, start)
    assert got["id"].size > 148 * 4 * 128
    for refill in (1, 32):
        want, wst = photons(gpu, p, grid, start, refill_threshold=refill)
        assert {k: st[k] for k in st if k != "trace_ms"} == {k: wst[k] for k in wst if k != "trace_ms"}
        for f in abi.PHOTON_FIELDS:
            assert np.array_equal(got[f].view(np.uint8), want[f].view(np.uint8)), (refill, f)
