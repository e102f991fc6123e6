"""Adam where it leaves cells alone: against its formula in 64 bits."""
import numpy as np
import pytest
import torch

import plenoxels_gb300 as pg

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _adam64(p, g, m, s, lr, b1, b2, eps, t):
    m = b1 * m.double() + (1 - b1) * g.double()
    s = b2 * s.double() + (1 - b2) * g.double() ** 2
    return p.double() - lr / (1 - b1 ** t) * m / (s.sqrt() / (1 - b2 ** t) ** 0.5 + eps), m, s


@pytest.mark.parametrize("dims", [(1, 1, 1), (7, 5, 3), (33, 64, 65), (150, 100, 90)])
@pytest.mark.parametrize("accumulate", [True, False])
def test_adam_on_a_sparse_gradient(dims, accumulate):
    gen = torch.Generator().manual_seed(7)
    p = torch.randn(*dims, 4, generator=gen)
    g = torch.randn(*dims, 4, generator=gen) * (torch.rand(*dims, 1, generator=gen) < 0.2)
    g[torch.rand(g.shape, generator=gen) < 0.3] = 0.0
    seen = torch.rand(*dims, 1, generator=gen) < 0.5
    m, s = torch.randn(p.shape, generator=gen) * seen, torch.rand(p.shape, generator=gen) * seen
    opt = pg.FusedAdam(p.to(DEV), 0.01, accumulate_abs_grad=accumulate)
    opt.exp_avg.copy_(m)
    opt.exp_avg_sq.copy_(s)
    if accumulate:
        opt.abs_grad.fill_(0.5)
    opt.step_count = 4
    grad = g.to(DEV)
    opt.step(grad)
    for got, want in zip((opt.grid, opt.exp_avg, opt.exp_avg_sq),
                         _adam64(p, g, m, s, 0.01, 0.9, 0.999, 1e-8, 5)):
        # four fp32 roundings of values up to a few units
        np.testing.assert_allclose(got.cpu().numpy(), want.numpy(), rtol=2e-6, atol=1e-6)
    rest = (~seen.expand_as(p)) & (g.abs().sum(-1, keepdim=True) == 0).expand_as(p)
    assert torch.equal(opt.grid.cpu()[rest], p[rest])
    assert not bool(grad.any())
    if accumulate:
        np.testing.assert_allclose(opt.abs_grad.cpu().numpy(), 0.5 + g.abs().numpy(), rtol=1e-6)


def test_adam_at_rest_keeps_nan_and_eps_zero_makes_it():
    p = torch.tensor([float("nan"), float("inf"), 1.0, -0.0], device=DEV).repeat(1, 1, 8, 1)
    opt = pg.FusedAdam(p.clone(), 0.01)
    grad = torch.zeros_like(p)
    grad[0, 0, 3, 1] = float("nan")
    opt.step(grad.clone(), zero_grad=False)
    rest = grad.abs().sum(-1, keepdim=True).expand_as(p) == 0
    np.testing.assert_array_equal(opt.grid[rest].cpu().numpy(), p[rest].cpu().numpy())
    assert bool(torch.isnan(opt.grid[0, 0, 3, 1])) and bool(torch.isnan(opt.abs_grad[0, 0, 3, 1]))
    opt = pg.FusedAdam(torch.ones_like(p), 0.01, eps=0.0)   # 0 / 0, as torch.optim.Adam
    opt.step(torch.zeros_like(p))
    assert bool(torch.isnan(opt.grid).all())
