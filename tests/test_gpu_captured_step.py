"""A FusedTrainStep with two gradient buffers in a CUDA graph: every replay and every step
beside it starts from a zero gradient."""
import pytest
import torch

import plenoxels_gb300 as pg

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("marked_cells", [0, 1 << 40])   # every grid marked, none marked
@pytest.mark.parametrize("steps", [1, 2, 3])
@pytest.mark.parametrize("warm_up", [2, 3])
def test_replays_start_from_a_zero_gradient(marked_cells, steps, warm_up, monkeypatch):
    monkeypatch.setattr(pg.render, "MARKED_CELLS", marked_cells)
    gen = torch.Generator(device=DEV).manual_seed(steps)
    grid = torch.rand(30, 31, 33, 4, generator=gen, device=DEV)
    grid[..., 3] *= 0.1
    args = (grid, 0.1, 90, 0.05)
    step = pg.FusedTrainStep(*args, overlap_zero=True, zeroing="marked")
    plain = pg.FusedTrainStep(*args)
    o, d, t = torch.empty(200, 3, device=DEV), torch.empty(200, 3, device=DEV), torch.empty(200, 4, device=DEV)

    def new_rays():
        o.copy_(torch.rand(200, 3, generator=gen, device=DEV) * 0.5 + torch.tensor([0.0, 0.0, 2.5], device=DEV))
        d.copy_(torch.nn.functional.normalize(torch.randn(200, 3, generator=gen, device=DEV) * 0.3
                                              - torch.tensor([0.0, 0.0, 1.0], device=DEV), dim=1))
        t.copy_(torch.rand(200, 4, generator=gen, device=DEV))

    def check(grad):
        plain.step_rays(o, d, t)
        assert float((grad - plain.grad).abs().max()) <= 1e-6 * float(plain.grad.abs().max())

    for _ in range(warm_up):
        new_rays()
        step.step_rays(o, d, t)
        check(step.grad)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        for _ in range(steps):
            step.step_rays(o, d, t)
    captured = step.grad
    for i in range(3):
        new_rays()
        graph.replay()
        check(captured)
        for _ in range(i):   # none, one, two steps beside the replays
            new_rays()
            step.step_rays(o, d, t)
            check(step.grad)
