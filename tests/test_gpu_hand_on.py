"""Warps that hand their last rays on to a second launch of the leg, on the ways
that trace besides one grt_run: a chunked step loop, the render graph, and
streamed renders, whose forward leg's fields are still on their way up while
the backward leg runs.  Images of more than five tiles for every warp, two
frequency channels to a geodesic; the photons bit for bit those of a run that
refills its warps early and hands nothing on."""

import numpy as np
import pytest

from grt import abi, workloads
from test_gpu_async import new_outs, pinned_block

pytestmark = pytest.mark.gpu

PX = 651


def scene(**kw):
    w = workloads.scaled(workloads.C2, pixels=PX, grid=(32, 16, 16), image_nx=PX, image_ny=PX, **kw)
    p = w.params()
    specs = [abi.ImageSpec.from_params(p, PX, PX, custom_frequency_hz=f, emission_coefficient=f / 2.3e11)
             for f in (2.3e11, 8.6e10)]
    return p, w.torus(), specs


def photons(ctx):
    ph = ctx.download_photons()
    return [getattr(ph, f).view(np.uint8) for f in abi.PHOTON_FIELDS]


@pytest.mark.parametrize("way", ["chunks", "graph", "async"])
def test_handed_on_rays_by_every_way(gpu, way):
    p, grid, specs = scene(**(dict(termination_percent=0.9, output_interval=9) if way == "chunks" else {}))
    with gpu.Context(p) as ctx:
        ctx.set_launch_config(refill_threshold=1)
        ctx.upload_grid(grid)
        ctx.init_image_batch(specs)
        start = pinned_block(ctx.n)
        ctx.download_photons(start)
        wstats = ctx.run()
        want = photons(ctx)
        wouts = ctx.all_batch_image_products(new_outs(p, specs))
    with gpu.Context(p) as ctx:
        ctx.upload_grid(grid)
        ctx.init_image_batch(specs)
        assert ctx.launch_config()["refill_threshold"] == 32 and -(-ctx.geodesics // 32) >= 5 * 148 * 4 * 4
        for _ in range(2):
            outs = new_outs(p, specs)
            if way == "chunks":
                ctx.init_image_batch(specs)
                stats = ctx.run()
            elif way == "graph":
                stats = ctx.render_graph()
            else:
                ctx.render_async(start, outs)
                stats = ctx.render_wait()
            if way != "async":
                ctx.all_batch_image_products(outs)
            for f, a, b in zip(abi.PHOTON_FIELDS, photons(ctx), want):
                assert np.array_equal(a, b), f
            for k in ("accepted_steps", "rejected_attempts", "photon_calls", "n_terminated", "steps_done"):
                assert stats[k] == wstats[k], k
            for a, b in zip(outs, wouts):
                # a pixel's arrivals add in any order
                assert np.allclose(a.image_I, b.image_I, rtol=1e-12, atol=0.0)
                assert int(a.arrived_count[0]) == int(b.arrived_count[0]) > 0
