"""The refill threshold the library picks while no launch shape is set (32 in
image mode, 4 in disk mode) changes no photon: against the thresholds at the
ends of the range, set by hand, with more rays than the resident lanes so that
warps do refill.  Images of more than five tiles for every resident warp also
hand the last rays of a tile on to a second launch at a threshold of 32; two
frequency channels that share their geodesics as well, and a run cut short by
its step count."""

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


@pytest.mark.parametrize("mode", ["image", "image_large", "image_cut", "channels", "disk"])
def test_default_refill_gives_the_same_photons(gpu, mode):
    if mode != "disk":
        px = 293 if mode == "image" else 651
        w = workloads.scaled(workloads.C2, pixels=px, grid=(32, 16, 16), image_nx=px, image_ny=px,
                             max_steps=27 if mode == "image_cut" else 4000,
                             precision=abi.PREC_MIXED if mode == "channels" else abi.PREC_FP64)
        p, grid = w.params(), w.torus()
        if mode == "channels":
            specs = [abi.ImageSpec.from_params(p, px, px, custom_frequency_hz=f, emission_coefficient=f / 2.3e11)
                     for f in (2.3e11, 8.6e10)]
            start = lambda ctx: ctx.init_image_batch(specs)  # noqa: E731
        else:
            start = lambda ctx: ctx.init_image_photons(px, px)  # noqa: E731
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
