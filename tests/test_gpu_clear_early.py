"""Launches with enough rays per warp that some warps begin with the clear of the other gradient
buffer: every step's gradient equals that of a step with a freshly zeroed one, and the other
buffer is zero after it."""
import numpy as np
import pytest
import torch

import plenoxels_gb300 as pg

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("mode,rays", [("trilinear", 18239), ("trilinear", 18240), ("trilinear", 40001),
                                       ("nearest", 24319), ("nearest", 24320), ("nearest", 50003)])
@pytest.mark.parametrize("dims", [(30, 31, 33), (150, 170, 163)])   # fewer rounds than blocks, more
@pytest.mark.parametrize("marked_cells", [0, 1 << 40])   # every grid marked, none marked
def test_steps_start_from_a_zero_gradient(mode, rays, dims, marked_cells, monkeypatch):
    monkeypatch.setattr(pg.render, "MARKED_CELLS", marked_cells)
    gen = torch.Generator(device=DEV).manual_seed(rays)
    grid = torch.rand(*dims, 4, generator=gen, device=DEV)
    grid[..., 3] *= 0.2
    pd, S = 3.0 / max(dims), 40
    a = pg.FusedTrainStep(grid, pd, S, 4.0 / S, mode=mode, overlap_zero=True, zeroing="marked")
    b = pg.FusedTrainStep(grid, pd, S, 4.0 / S, mode=mode)
    for _ in range(3):
        o = torch.randn(rays, 3, generator=gen, device=DEV) * 0.3 + torch.tensor([0.0, 0.0, 3.5], device=DEV)
        d = torch.nn.functional.normalize(torch.randn(rays, 3, generator=gen, device=DEV) * 0.3
                                          - torch.tensor([0.0, 0.0, 1.0], device=DEV), dim=1)
        t = torch.rand(rays, 4, generator=gen, device=DEV)
        la, lb = a.step_rays(o, d, t), b.step_rays(o, d, t)
        np.testing.assert_array_equal(la.cpu().numpy(), lb.cpu().numpy())
        # the rays' updates of a cell come in any order
        assert float((a.grad - b.grad).abs().max()) <= 1e-5 * float(b.grad.abs().max())
        assert not bool(a._grads[1 - a._buf].any())
        assert a._marks is None or not bool(a._marks[1 - a._buf].any())
