"""The render kernel's clear of the other gradient buffer: every step's gradient equals that
of a step with a freshly zeroed one, whatever the number of rays, cells and marked units."""
import numpy as np
import pytest
import torch

import plenoxels_gb300 as pg
from plenoxels_gb300 import _lib
from plenoxels_gb300._lib import ptr

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rays(n, gen, dtype):
    o = torch.randn(n, 3, generator=gen, device=DEV) * 0.3 + torch.tensor([0.0, 0.0, 3.5], device=DEV)
    d = torch.nn.functional.normalize(torch.randn(n, 3, generator=gen, device=DEV) * 0.3
                                      - torch.tensor([0.0, 0.0, 1.0], device=DEV), dim=1)
    return o.to(dtype), d.to(dtype), torch.rand(n, 4, generator=gen, device=DEV).to(dtype)


@pytest.mark.parametrize("dims,rays", [((3, 5, 7), 40), ((33, 40, 31), 1), ((33, 40, 31), 3000),
                                       ((130, 127, 129), 5), ((64, 64, 64), 20000)])
@pytest.mark.parametrize("mode", ["nearest", "trilinear"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("marked_cells", [0, 1 << 40])   # every grid marked, none marked
def test_steps_start_from_a_zero_gradient(dims, rays, mode, dtype, marked_cells, monkeypatch):
    monkeypatch.setattr(pg.render, "MARKED_CELLS", marked_cells)
    gen = torch.Generator(device=DEV).manual_seed(rays)
    grid = torch.rand(*dims, 4, generator=gen, device=DEV, dtype=dtype)
    grid[..., 3] *= 0.2
    pd, S = 3.0 / max(dims), 70
    a = pg.FusedTrainStep(grid, pd, S, 4.0 / S, mode=mode, overlap_zero=True, zeroing="marked")
    b = pg.FusedTrainStep(grid, pd, S, 4.0 / S, mode=mode)
    for i in range(5):
        o, d, t = _rays(rays if i != 2 else 0, gen, dtype)
        zero = i != 3   # one step accumulates
        la, lb = a.step_rays(o, d, t, zero_grad=zero), b.step_rays(o, d, t, zero_grad=zero)
        np.testing.assert_array_equal(la.cpu().numpy(), lb.cpu().numpy())
        scale = float(b.grad.abs().max())
        assert float((a.grad - b.grad).abs().max()) <= 1e-6 * scale
    other = a._grads[1 - a._buf]
    assert not bool(other.any())
    assert a._marks is None or not bool(a._marks[1 - a._buf].any())


def test_arguments(monkeypatch):
    monkeypatch.setattr(pg.render, "MARKED_CELLS", 0)
    grid = torch.rand(4, 4, 4, 4, device=DEV)
    step = pg.FusedTrainStep(grid, 0.5, 8, 0.5, overlap_zero=True, zeroing="marked")
    gd = _lib.make_grid(grid, step.grid_min, 0.5, step.mode, True)
    rd = _lib.PgbRays(num_rays=0, num_samples=8, delta_step=0.5, grad_marks=ptr(step._marks[0]))
    terms = _lib.PgbLossTerms(1.0, 0.0, 1e-4)
    call = _lib.load().pgb_render_train_clear
    g0, g1, m0, m1 = (ptr(t) for t in (*step._grads, *step._marks))
    head = (gd, rd, None, terms, None)
    assert call(*head, g0, ptr(step.losses), ptr(step.workspace), g0, m1, 0) == _lib.PGB_ERR_ARG
    assert call(*head, g0, ptr(step.losses), ptr(step.workspace), g1, m0, 0) == _lib.PGB_ERR_ARG
    assert call(*head, g0, ptr(step.losses), ptr(step.workspace), None, m1, 0) == _lib.PGB_ERR_ARG
    assert call(*head, g0, ptr(step.losses), ptr(step.workspace), g0, None, 0) == _lib.PGB_ERR_ARG
    assert call(*head, g0, ptr(step.losses), ptr(step.workspace), g1 + 4, m1, 0) == _lib.PGB_ERR_ALIGN
