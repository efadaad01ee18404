"""The step loop with termination_percent < 1 enqueues several chunks at a time
and stops on the device.  Against the oracle's loop, which looks after every
output step: the same photons, step count and terminated count whether the
fraction is reached in the first chunk, in the middle of a batch of chunks,
across batches or never, for whole-ray and split chunks."""

import pytest

from grt import workloads
from helpers import assert_photons_match, mini, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interval", [1, 3, 5])
@pytest.mark.parametrize("fraction", [0.01, 0.5, 0.9, 0.999999])
@pytest.mark.parametrize("split", [None, 0, 1])
def test_chunked_loop_stops_where_the_reference_stops(gpu, oracle, interval, fraction, split):
    w = mini(workloads.C2, 14, (24, 16, 16), termination_percent=fraction, output_interval=interval, max_steps=60)
    p, grid = w.params(), w.torus()
    launch = None if split is None else dict(split_legs=split)
    got, _, gst = run_gpu(gpu, p, grid, nx=14, ny=14, launch=launch)
    want, _, wst = run_oracle(oracle, p, grid, nx=14, ny=14)
    assert_photons_match(got, want)
    assert (gst["steps_done"], gst["n_terminated"]) == (wst["steps_done"], wst["n_terminated"])


@pytest.mark.parametrize("interval,max_steps", [(1, 5), (1, 16), (1, 17), (2, 33), (7, 8)])
def test_a_loop_that_runs_out_of_steps(gpu, oracle, interval, max_steps):
    w = mini(workloads.C2, 10, (24, 16, 16), termination_percent=0.95, output_interval=interval, max_steps=max_steps)
    p, grid = w.params(), w.torus()
    got, _, gst = run_gpu(gpu, p, grid, nx=10, ny=10)
    want, _, wst = run_oracle(oracle, p, grid, nx=10, ny=10)
    assert_photons_match(got, want)
    assert (gst["steps_done"], gst["n_terminated"]) == (wst["steps_done"], wst["n_terminated"])
