"""The pooled gradient's update in one pass, and pooling by strides, against F.avg_pool3d and
the two separate passes."""
import numpy as np
import pytest
import torch

import plenoxels_gb300 as pg
from plenoxels_gb300.grid_functions import pool_shape

pytestmark = pytest.mark.gpu
DEV = "cuda"


WINDOWS = [(3, 1), (7, 1), (8, 1), (9, 1), (9, 2), (16, 8), (21, 5), (45, 11), (5, 5), (2, 7), (19, 1)]


@pytest.mark.parametrize("window,stride", WINDOWS)
@pytest.mark.parametrize("dims", [(45, 46, 47), (61, 50, 200)])
def test_pool_and_pooled_update(window, stride, dims):
    gen = torch.Generator(device=DEV).manual_seed(window * 100 + stride)
    grid = torch.randn(*dims, 4, generator=gen, device=DEV)
    out = pg.average_pool3d_grid(grid, window, stride)
    ref = torch.nn.functional.avg_pool3d(grid.double().permute(3, 0, 1, 2)[None], (window,) * 3,
                                         stride=stride)[0].permute(1, 2, 3, 0)
    # three sums of at most 45 fp32 terms of magnitude up to about 5, then the division
    np.testing.assert_allclose(out.cpu().numpy(), ref.cpu().numpy(), rtol=0, atol=3 * 45 * 5 * 2.0 ** -24)
    d_out = torch.randn(out.shape, generator=gen, device=DEV)
    x = grid.clone().requires_grad_(True)
    pg.average_pool3d_grid(x, window, stride).backward(d_out)
    _, nbytes = pool_shape(dims + (4,), window, stride)
    scratch = torch.empty(max(16, nbytes), dtype=torch.uint8, device=DEV)
    a, b = pg.FusedAdam(grid.clone(), 0.01), pg.FusedAdam(grid.clone(), 0.01)
    for _ in range(2):
        a.step(x.grad.clone())
        b.step_pooled(d_out, window, stride, scratch)
    for u, v in ((a.grid, b.grid), (a.exp_avg, b.exp_avg), (a.exp_avg_sq, b.exp_avg_sq), (a.abs_grad, b.abs_grad)):
        # the same arithmetic up to fused roundings, on values of at most a few units
        np.testing.assert_allclose(u.cpu().numpy(), v.cpu().numpy(), rtol=1e-6, atol=1e-7)


def test_trainer_keeps_the_rules_of_a_written_full_gradient():
    """A caller's write to the full gradient is overwritten and zeroed by a pooled step."""
    gen = torch.Generator(device=DEV).manual_seed(3)
    grid = torch.rand(40, 40, 40, 4, generator=gen, device=DEV) * 0.2
    o = torch.tensor([0.0, 0.0, 4.0], device=DEV).repeat(64, 1)
    d = torch.nn.functional.normalize(torch.randn(64, 3, generator=gen, device=DEV) * 0.1
                                      - torch.tensor([0.0, 0.0, 1.0], device=DEV), dim=1)
    t = torch.rand(64, 4, generator=gen, device=DEV)
    runs = []
    for write in (False, True):
        tr = pg.Trainer(grid.clone(), 3.0 / 40, 64, 4.0 / 64, 0.01, tv=1e-3, progressive_growing=True,
                        fields=[9, 5], steps_per_field=1)
        for i in range(3):
            if write and i < 2:
                tr.render.grad.fill_(7.0)
            tr.step_rays(o, d, t)
            assert not bool(tr.render.grad.any())
        runs.append(tr)
    np.testing.assert_allclose(runs[0].grid.cpu().numpy(), runs[1].grid.cpu().numpy(), rtol=1e-5, atol=1e-6)
