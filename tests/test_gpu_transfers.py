"""Products and gradients by the different ways they leave the device: the image
products through the pinned stage, straight into ordinary arrays or into
page-locked ones, against the products block of the same photons; the
differentiable render on device tensors against host arrays."""

import numpy as np
import pytest

from grt import abi, torus, workloads

pytestmark = pytest.mark.gpu


# 4 nx ny + bins + 1 values: the smallest, odd planes, the largest block of the stage (81,920) and one more, larger ones
@pytest.mark.parametrize("nx,ny,bins", [(1, 1, 1), (1, 3, 2), (37, 19, 128), (91, 90, 7), (128, 64, 1), (128, 64, 128), (128, 128, 1), (143, 143, 123), (143, 143, 124),
                                        (181, 181, 3), (131, 77, 5), (300, 211, 64)])
def test_image_products_by_every_way_out(gpu, nx, ny, bins):
    import torch
    w = workloads.scaled(workloads.C2, pixels=nx, grid=(24, 16, 16), image_nx=nx, image_ny=ny, spectrum_bins=bins,
                         spectrum_min_hz=1e10, spectrum_max_hz=1e13)
    p = w.params()
    with gpu.Context(p) as ctx:
        ctx.upload_grid(w.torus())
        ctx.init_image_photons(nx, ny)
        ctx.run()
        block = torch.empty(ctx.products_block_bytes // 8, dtype=torch.float64)
        ctx.copy_products_block(block.data_ptr(), block.numel() * 8)
        ctx.synchronize()
        block = block.numpy()
        pinned = abi.ProductArrays.for_params(p)
        for f in ("image_I", "image_Q", "image_U", "image_V"):
            setattr(pinned, f, torch.full((ny, nx), 7.0, dtype=torch.float64, pin_memory=True).numpy())
        for out in (ctx.image_products(), ctx.image_products(pinned), ctx.image_products(abi.ProductArrays.for_params(p))):
            for q, f in enumerate(("image_I", "image_Q", "image_U", "image_V")):
                # a pixel's arrivals add in any order
                assert np.allclose(getattr(out, f).ravel(), block[q * nx * ny:(q + 1) * nx * ny], rtol=1e-12, atol=0.0)
            assert np.allclose(out.spectrum_I, block[4 * nx * ny:4 * nx * ny + bins], rtol=1e-12, atol=0.0)
            assert int(out.arrived_count[0]) == int(block[-1:].view(np.uint64)[0]) > 0


@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_render_on_the_device_equals_host_arrays(gpu, dtype):
    import torch
    from grt.autograd import ImageRenderer
    w = workloads.scaled(workloads.C4, pixels=24, grid=(32, 16, 16), image_nx=24, image_ny=24)
    p, grid = w.params(), torus.benchmark_torus(32, 16, 16, spin=0.9)
    rng = np.random.default_rng(3)
    host = [torch.from_numpy(np.exp(rng.normal(0, 0.1, (32, 16, 16)))).to(getattr(torch, dtype)) for _ in range(2)]
    weights = torch.from_numpy(rng.normal(size=(24, 24))).to(getattr(torch, dtype))
    r = ImageRenderer(p, grid)
    got = []
    for device in ("cpu", "cuda"):
        m = [t.to(device).clone().requires_grad_(True) for t in host]
        image = r.render(*m)
        assert image.device.type == device and image.dtype == m[0].dtype
        # a broadcast gradient too: not contiguous
        grads = torch.autograd.grad((image * weights.to(device)).sum(), m, retain_graph=True)
        flat = torch.autograd.grad(image.sum(), m)
        got.append([t.detach().cpu().double().numpy() for t in (image, *grads, *flat)])
    tol = 1e-12 if dtype == "float64" else 2.0 ** -23
    for a, b in zip(*got):
        assert np.abs(a - b).max() <= tol * np.abs(a).max()
    # a transposed multiplier is laid out first
    t = torch.from_numpy(np.ascontiguousarray(host[0].numpy().T)).to("cuda").permute(2, 1, 0)
    image = r.render(t, host[1].to("cuda"))
    assert np.abs(image.cpu().double().numpy() - got[1][0]).max() <= tol * np.abs(got[1][0]).max()
    r.close()
