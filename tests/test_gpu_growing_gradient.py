"""Progressive growing with a full gradient that something else writes between the steps: the
training loop's results are those of a run in which nothing did."""
import numpy as np
import pytest
import torch

import plenoxels_gb300 as pg

pytestmark = pytest.mark.gpu
DEV = "cuda"

WRITES = {
    "a loss on the full grid": lambda tr, o, d, t: tr.render.step_rays(o, d, t),
    "a loss on the full grid, accumulated": lambda tr, o, d, t: tr.render.step_rays(o, d, t, zero_grad=False),
    "a TV gradient": lambda tr, o, d, t: tr.opt.add_tv(tr.render.grad, 1.0),
    "an operator": lambda tr, o, d, t: tr.render.grad.add_(1.0),
    "past torch's counter": lambda tr, o, d, t: tr.render.grad.data.fill_(1.0),
}


@pytest.mark.parametrize("write", WRITES)
@pytest.mark.parametrize("tv", [0.0, 1e-3])
@pytest.mark.parametrize("jump", [False, True])   # from a receptive field straight to the full grid
def test_written_full_gradient_does_not_reach_a_step(write, tv, jump):
    gen = torch.Generator(device=DEV).manual_seed(3)
    grid = torch.rand(40, 41, 39, 4, generator=gen, device=DEV) * 0.2
    o = torch.tensor([0.0, 0.0, 4.0], device=DEV).repeat(64, 1)
    d = torch.nn.functional.normalize(torch.randn(64, 3, generator=gen, device=DEV) * 0.1
                                      - torch.tensor([0.0, 0.0, 1.0], device=DEV), dim=1)
    t = torch.rand(64, 4, generator=gen, device=DEV)
    runs = []
    for written in (False, True):
        tr = pg.Trainer(grid.clone(), 3.0 / 41, 64, 4.0 / 64, 0.01, tv=tv, progressive_growing=True,
                        fields=[9, 7, 5], steps_per_field=1)
        for _ in range(4):
            growing = tr.field(tr.step_index) > 1
            if written and growing:
                WRITES[write](tr, o, d, t)
            tr.step_rays(o, d, t)
            if jump and growing:
                tr.step_index = 3
            if write != "past torch's counter" or tr.field(tr.step_index) <= 1 and not jump:
                assert not bool(tr.render.grad.any())
        runs.append(tr)
    # the rays' float atomics come in any order, which Adam's quotient of moments shows in cells
    # whose gradient nearly cancels: sums of |gradient| to rounding, the grid on average
    a, b = runs
    np.testing.assert_allclose(b.opt.abs_grad.cpu().numpy(), a.opt.abs_grad.cpu().numpy(), rtol=1e-3, atol=1e-5)
    assert float((a.grid - b.grid).abs().mean()) <= 1e-5


def test_trainer_made_in_inference_mode():
    """Such a trainer's tensors have no version counter."""
    gen = torch.Generator(device=DEV).manual_seed(4)
    grid = torch.rand(24, 25, 23, 4, generator=gen, device=DEV) * 0.2
    o = torch.tensor([0.0, 0.0, 4.0], device=DEV).repeat(64, 1)
    d = torch.nn.functional.normalize(torch.randn(64, 3, generator=gen, device=DEV) * 0.1
                                      - torch.tensor([0.0, 0.0, 1.0], device=DEV), dim=1)
    t = torch.rand(64, 4, generator=gen, device=DEV)
    runs = []
    for inference in (False, True):
        with torch.inference_mode(inference):
            tr = pg.Trainer(grid.clone(), 3.0 / 25, 64, 4.0 / 64, 0.01, tv=1e-3, progressive_growing=True,
                            fields=[9, 5], steps_per_field=1)
            for i in range(3):
                if inference and i < 2:
                    tr.render.grad.fill_(1.0)
                    tr.opt.add_tv(tr.render.grad, 1.0)
                tr.step_rays(o, d, t)
                assert not bool(tr.render.grad.any())
        runs.append(tr)
    np.testing.assert_allclose(runs[1].opt.abs_grad.cpu().numpy(), runs[0].opt.abs_grad.cpu().numpy(),
                               rtol=1e-3, atol=1e-5)
