"""Host code of the C ABI where a call fails or a buffer does not fit, without a
GPU: csrc/grt_api.cu and grt_host.cpp compiled against stand-ins for the CUDA
runtime and the kernel launches (fake_cuda/fake_cuda.cpp)."""

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from grt import abi, autotune, lib, torus, workloads

HERE = Path(__file__).resolve().parent
SRC = HERE.parent / "gr-ray-tracer_b200" / "csrc"
GRID = (8, 6, 5)


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    out = tmp_path_factory.mktemp("fake") / "libgrt_fake.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I/usr/local/cuda/include",
                    f"-I{SRC}", f"-I{HERE.parent / 'include'}", "-x", "c++", str(SRC / "grt_api.cu"),
                    str(SRC / "grt_host.cpp"), str(HERE / "fake_cuda" / "fake_cuda.cpp"), "-o", str(out)], check=True)
    return out


@pytest.fixture
def fake(built, monkeypatch):
    monkeypatch.setattr(lib, "_lib", None)
    L = lib.load(built)
    L.fake_reset.argtypes = L.fake_limit.argtypes = L.fake_malloc.argtypes = [C.c_size_t]
    L.fake_used.restype = C.c_size_t
    L.fake_malloc.restype = C.c_void_p
    L.fake_launches.restype = C.c_char_p
    L.fake_reset(1 << 34)
    yield L
    assert L.fake_bad_accesses() == 0


def image(px, **kw):
    return workloads.scaled(workloads.C2, pixels=px, grid=GRID, image_nx=px, image_ny=px).params().update(**kw)


def fluid():
    return torus.benchmark_torus(*GRID, spin=workloads.C2.spin)


def launches(fake, what=""):
    return [line for line in fake.fake_launches().decode().splitlines() if line.startswith(what)]


class DeviceArray:
    """What Context asks of a CUDA tensor: a contiguous float64 one of the given shape."""
    is_cuda, dtype = True, "torch.float64"

    def __init__(self, fake, *shape):
        self.shape = shape
        self._ptr = fake.fake_malloc(8 * self.numel())

    def is_contiguous(self):
        return True

    def numel(self):
        return int(np.prod(self.shape))

    def data_ptr(self):
        return self._ptr


@pytest.mark.parametrize("directory", [False, True])
def test_buffers_shorter_than_the_grid_are_refused(fake, tmp_path, directory):
    p, grid, cells = image(4), fluid(), int(np.prod(GRID))
    with lib.Context(p) as ctx:
        if directory:
            for k in torus.FIELD_FILES:
                np.save(tmp_path / k, grid[k])
            ctx.upload_grid_numpy_dir(tmp_path)
        else:
            ctx.upload_grid(grid)
        whole, short = DeviceArray(fake, *GRID), DeviceArray(fake, cells - 1)
        for pair in ((short, None), (None, short), (whole, short), (np.ones(cells - 1), None), (np.ones(()), None)):
            with pytest.raises(ValueError, match="cells"):
                ctx.set_cell_multipliers(*pair)
        ctx.set_cell_multipliers(whole, np.ones(GRID))
        ctx.init_image_forward_photons(4, 4, 60.0)
        ctx.forward_checkpointed(8)
        dL = DeviceArray(fake, 4, 4)
        for pair in ((short, whole), (whole, short)):
            with pytest.raises(ValueError, match="cells"):
                ctx.adjoint_image_I_device(dL, *pair)
        with pytest.raises(ValueError, match="cells"):
            ctx.adjoint_image_I(np.zeros((4, 4)), (cells - 1,))
        ctx.adjoint_image_I_device(dL, whole, DeviceArray(fake, cells))
        assert ctx.adjoint_image_I(np.zeros((4, 4)), GRID)[0].shape == GRID


@pytest.mark.parametrize("what", ["random", "pixels", "batch", "upload", "disk"])
def test_a_failed_initialisation_leaves_no_photons(fake, what):
    """... so that no later call traces the photons, images or queue order of the set before it."""
    p = image(10)
    with lib.Context(p) as ctx:
        ctx.upload_grid(fluid())
        ctx.init_image_photons(10, 10)
        ctx.run()
        assert launches(fake, "trace 1")[-1].split("order=")[1] == "99"
        if what in ("random", "pixels"):
            fake.fake_fail_init(1)
        else:
            fake.fake_limit(fake.fake_used())
        with pytest.raises(lib.GrtError):
            if what == "random":
                ctx.init_image_photons_random(50)
            elif what == "pixels":
                ctx.init_image_photons(5, 5)
            elif what == "batch":
                ctx.init_image_batch([abi.ImageSpec.from_params(p, 5, 5)] * 2)
            elif what == "upload":
                ctx.upload_photons(abi.PhotonArrays(101))
            else:
                ctx.init_disk_photons()
        fake.fake_reset(1 << 34)
        assert ctx.n == 0 and ctx.run()["n_terminated"] == 0 and not launches(fake, "trace")
        with pytest.raises(lib.GrtError):
            ctx.render_graph()
        # and the next one starts afresh
        ctx.init_image_photons_random(50)
        ctx.run()
        ctx.init_image_photons(10, 10)
        ctx.run()
        assert [line.split("order=")[1] for line in launches(fake, "trace 1")] == ["49", "99"]


@pytest.mark.parametrize("separable,norm,blocks", [(True, 500.0, 2), (False, 500.0, 4), (False, 2.0, 2)])
def test_disk_blocks_by_the_grid(fake, separable, norm, blocks):
    """Two or three blocks a multiprocessor are enough where a sample is a few reads of the axes; the scans of a grid
    that is not separable want every packet resident that can be."""
    w = workloads.DiskWorkload("disk", (24, 16, 16), 0.9, norm)
    grid = torus.benchmark_torus(*w.grid, spin=w.spin)
    if not separable:
        grid = dict(grid, **{"theta.npy": grid["theta.npy"] + 1e-4 * np.sin(grid["r.npy"])})
    with lib.Context(w.params()) as ctx:
        ctx.upload_grid(grid)
        n = ctx.init_disk_photons()
        assert n <= 148 * 2 * 128 if norm < 100 else 148 * 3 * 128 < n <= 8 * 2 * 148 * 128
        ctx.run()
    (line,) = launches(fake, "trace 3")
    assert f"blocks={blocks} " in line


def differentiate(fake, ctx, px, squeeze=False):
    """The calls of one differentiable render; with squeeze, no memory is left once the forward pass has returned."""
    ctx.set_cell_multipliers(np.ones(GRID), np.ones(GRID))
    ctx.init_image_forward_photons(px, px, 60.0)
    ctx.forward_checkpointed(64)
    held = fake.fake_used()
    if squeeze:
        fake.fake_limit(held)
    ctx.image_products()
    ctx.adjoint_image_I(np.ones((px, px)), GRID)
    return held


def test_the_record_of_updates_leaves_memory_to_what_is_needed(fake):
    px = 40
    record = px * px * 128 * 48
    with lib.Context(image(px)) as ctx:
        ctx.upload_grid(fluid())
        differentiate(fake, ctx, px)
        assert launches(fake, "forward") == ["forward cap=128"] and launches(fake, "sweep") == ["sweep"]
        needed = fake.fake_used() - record
    # room for all but the record: rays are traced again
    for memory in (needed, needed + record // 2):
        fake.fake_reset(memory)
        with lib.Context(image(px)) as ctx:
            ctx.upload_grid(fluid())
            differentiate(fake, ctx, px)
            assert launches(fake, "forward") == ["forward cap=0"]
    # a record that is there goes when another buffer needs the room, in the
    # same render and in a larger one after it
    fake.fake_reset(1 << 34)
    with lib.Context(image(px)) as ctx:
        ctx.upload_grid(fluid())
        held = differentiate(fake, ctx, px, squeeze=True)
        assert launches(fake, "forward") == ["forward cap=128"]
        assert launches(fake, "reverse") and not launches(fake, "sweep")
        assert fake.fake_used() <= held - record // 2
        fake.fake_reset(1 << 34)
        differentiate(fake, ctx, px)
        fake.fake_limit(fake.fake_used())
        ctx.init_image_photons(2 * px, px)  # 146 bytes a photon where the record held 6144
        ctx.init_image_photons_random(px * px)
        ctx.run()


def test_products_without_memory_to_pin_are_copied_directly(fake):
    with lib.Context(image(16)) as ctx:
        ctx.upload_grid(fluid())
        ctx.init_image_photons(16, 16)
        ctx.run()
        fake.fake_refuse_pinned(1)
        ctx.image_products()
        fake.fake_refuse_pinned(0)
        ctx.image_products()


@pytest.mark.parametrize("field", ["image_I", "image_Q", "spectrum_I", "arrived_count"])
def test_device_memory_as_a_product_array_is_an_error(fake, field):
    """... and not written by the host, whichever array it is."""
    with lib.Context(image(16)) as ctx:
        ctx.upload_grid(fluid())
        ctx.init_image_photons(16, 16)
        ctx.run()
        arrays = abi.ProductArrays.for_params(ctx.params)
        out = arrays.struct()
        ptr = DeviceArray(fake, 16, 16).data_ptr()
        C.memset(ptr, 7, 16 * 16 * 8)
        setattr(out, field, C.cast(ptr, type(getattr(out, field))))
        assert fake.grt_get_image_products(ctx.handle, C.byref(out)) == abi.GRT_ECUDA
        assert C.string_at(ptr, 16 * 16 * 8) == b"\7" * (16 * 16 * 8)


def thresholds(fake):
    return [int(line.split("refill=")[1].split()[0]) for line in launches(fake, "trace")]


def test_a_field_of_the_launch_shape_leaves_the_refill_threshold_to_the_mode(fake):
    disk = workloads.DiskWorkload("disk", GRID, 0.9, 500.0).params()
    with lib.Context(image(700)) as ctx:
        ctx.upload_grid(fluid())
        assert ctx.launch_config()["refill_threshold"] == 32
        ctx.set_launch_config(max_iterations=10**9)  # gets, changes one field, sets
        ctx.init_image_photons(700, 700)
        ctx.run()
        assert set(thresholds(fake)) == {32}
        assert [line.split()[1] for line in launches(fake, "trace") if "hands_on" in line] == ["1", "2"]
        fake.fake_clear()
        ctx.set_params(disk)
        assert ctx.launch_config()["refill_threshold"] == 4
        ctx.init_disk_photons()
        ctx.run()
        assert thresholds(fake) == [4]
        fake.fake_clear()
        ctx.set_launch_config(refill_threshold=8)  # a threshold of the caller's own stays
        ctx.run()
        ctx.set_params(image(700))
        ctx.init_image_photons(700, 700)
        ctx.run()
        assert set(thresholds(fake)) == {8} and not any("hands_on" in line for line in launches(fake, "trace"))
        assert ctx.launch_config()["refill_threshold"] == 8


def test_the_tuner_keeps_the_shape_in_force_when_nothing_is_faster(monkeypatch):
    monkeypatch.setattr(autotune, "_CACHE", {})
    own = dict(threads_per_block=128, blocks_per_sm=0, refill_threshold=4, photons_per_grab=32, split_legs=1,
               max_iterations=0)

    class Tuned:
        params = workloads.DiskWorkload("disk", GRID, 0.9, 2.0).params()
        shape = dict(own)

        def launch_config(self):
            return dict(self.shape)

        def set_launch_config(self, **kw):
            self.shape.update(kw)

        def run(self):
            return dict(trace_ms=1.0 if self.shape["blocks_per_sm"] == 0 else 2.0)

    ctx = Tuned()
    best, ms, table = autotune.tune(ctx, lambda c: None, "disk")
    assert best == own == ctx.shape and ms == 1.0 and len(table) == 1 + len(list(autotune.candidates(False)))


def test_multipliers_go_with_a_grid_of_other_cells(fake):
    with lib.Context(image(4)) as ctx:
        ctx.upload_grid(fluid())
        ctx.set_cell_multipliers(np.ones(GRID), np.ones(GRID))
        ctx.upload_grid(fluid())  # as many cells: they stay
        ctx.init_image_photons(4, 4)
        ctx.run()
        assert launches(fake, "multipliers")
        fake.fake_clear()
        ctx.upload_grid(torus.benchmark_torus(16, 12, 10, spin=workloads.C2.spin))
        ctx.init_image_photons(4, 4)
        ctx.run()
        assert launches(fake, "trace") and not launches(fake, "multipliers")


@pytest.mark.parametrize("way", ["run", "graph", "async"])
def test_each_leg_hands_on_to_a_second_launch(fake, way):
    """... which belongs to the leg in the statistics, and comes before what waits for the photons' late fields."""
    p = image(700)
    specs = [abi.ImageSpec.from_params(p, 700, 700)]
    with lib.Context(p) as ctx:
        ctx.upload_grid(fluid())
        ctx.init_image_batch(specs)
        fake.fake_clear()
        if way == "async":
            ctx.render_async(abi.PhotonArrays.block(ctx.n), [abi.ProductArrays(700, 700, p.spectrum_bins)])
            stats = ctx.render_wait()
        else:
            stats = ctx.run() if way == "run" else ctx.render_graph()
    steps = [" ".join(line.split()[:2] + [w for w in line.split() if w in ("hands_on", "resume")])
             for line in launches(fake)]
    legs = [s for s in steps if s.startswith("trace") or s == "generate"]
    assert legs == ["trace 1 hands_on", "trace 1 resume", "generate", "trace 2 hands_on", "trace 2 resume"]
    assert stats["launches"] == 3
    if way == "async":
        assert steps[steps.index("trace 1 resume") + 1] == "wait" and steps.index("wait") < steps.index(legs[0])
