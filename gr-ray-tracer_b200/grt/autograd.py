"""torch.autograd.Function over the C ABI's differentiable radiative transfer.

ImageRenderer holds one device context (grid uploaded, camera from the
params).  render(m_abs, m_emis) returns the Stokes-I image as a torch tensor
whose backward is the hand-written adjoint kernel (grt_adjoint_image_I):
forward = grt_set_cell_multipliers + grt_init_image_forward_photons
(line-of-sight rays through the fluid) + grt_forward_checkpointed +
grt_get_image_products; backward = the adjoint
sweep.  Multipliers, image and gradients on the device stay there: the library
reads and writes the tensors' memory (through host arrays the four copies of a
128 x 128 image on a 96 x 48 x 48 grid took as long as the trace).  Nothing is
computed in torch except the loss the caller builds on the returned image.
"""

from __future__ import annotations

import numpy as np
import torch

from . import lib


class ImageRenderer:
    def __init__(self, params, grid: dict, checkpoint_interval: int = 64, back_distance: float = 60.0):
        self.ctx = lib.Context(params)
        self.ctx.upload_grid(grid)
        self.grid_shape = tuple(grid["r.npy"].shape)
        self.params = params
        self.K = int(checkpoint_interval)
        self.back = float(back_distance)
        self.last_stats = None

    def close(self):
        self.ctx.close()

    def forward_image(self, m_abs: np.ndarray, m_emis: np.ndarray) -> np.ndarray:
        self.ctx.set_cell_multipliers(m_abs, m_emis)
        self.ctx.init_image_forward_photons(self.params.image_nx, self.params.image_ny, self.back)
        self.last_stats = self.ctx.forward_checkpointed(self.K)
        return self.ctx.image_products().image_I.copy()

    def backward_image(self, dL_dI: np.ndarray):
        return self.ctx.adjoint_image_I(dL_dI, self.grid_shape)

    # the same on the device: float64 CUDA tensors in and out
    def _forward_device(self, m_abs: torch.Tensor, m_emis: torch.Tensor) -> torch.Tensor:
        ny, nx = int(self.params.image_ny), int(self.params.image_nx)
        block = torch.empty(4 * ny * nx + int(self.params.spectrum_bins) + 1, dtype=torch.float64, device=m_abs.device)
        # the context has a stream of its own: what torch enqueued on this
        # memory comes first, and the image is complete before torch goes on
        torch.cuda.current_stream(m_abs.device).synchronize()
        self.ctx.set_cell_multipliers(m_abs, m_emis)
        self.ctx.init_image_forward_photons(nx, ny, self.back)
        self.last_stats = self.ctx.forward_checkpointed(self.K)
        self.ctx.copy_products_block(block.data_ptr(), block.numel() * 8)
        self.ctx.synchronize()
        return block[:ny * nx].view(ny, nx)

    def _backward_device(self, dL_dI: torch.Tensor):
        ga, ge = (torch.empty(self.grid_shape, dtype=torch.float64, device=dL_dI.device) for _ in range(2))
        torch.cuda.current_stream(dL_dI.device).synchronize()
        self.ctx.adjoint_image_I_device(dL_dI, ga, ge)
        return ga, ge

    def render(self, m_abs: torch.Tensor, m_emis: torch.Tensor) -> torch.Tensor:
        return _RenderStokesI.apply(m_abs, m_emis, self)


def _on_device(t: torch.Tensor, shape) -> bool:
    return t.is_cuda and tuple(t.shape) == tuple(shape)


class _RenderStokesI(torch.autograd.Function):
    @staticmethod
    def forward(ctx, m_abs, m_emis, renderer):
        ctx.renderer = renderer
        ctx.dtype = m_abs.dtype
        ctx.device = m_abs.device
        if all(_on_device(m, renderer.grid_shape) for m in (m_abs, m_emis)):
            img = renderer._forward_device(*(m.detach().double().contiguous() for m in (m_abs, m_emis)))
            return img.to(device=m_abs.device, dtype=m_abs.dtype, copy=True)
        img = renderer.forward_image(m_abs.detach().double().cpu().numpy(),
                                     m_emis.detach().double().cpu().numpy())
        return torch.from_numpy(img).to(device=m_abs.device, dtype=m_abs.dtype)

    @staticmethod
    def backward(ctx, grad_img):
        to = dict(device=ctx.device, dtype=ctx.dtype)
        if grad_img.is_cuda:
            ga, ge = ctx.renderer._backward_device(grad_img.detach().double().contiguous())
            return ga.to(**to), ge.to(**to), None
        ga, ge = ctx.renderer.backward_image(grad_img.detach().double().cpu().numpy())
        return torch.from_numpy(ga).to(**to), torch.from_numpy(ge).to(**to), None
