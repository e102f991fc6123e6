"""The gradient of a nearest ray without early stop does not depend on whether its chunks of 64
samples are picked by the library or asked for."""
import pytest
import torch

import plenoxels_gb300 as pg

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("samples", [64, 128, 129, 200, 600])
@pytest.mark.parametrize("kw", [dict(beta=5e-3), dict(clip=False), {}], ids=["beta", "no clip", "early stop"])
def test_picked_and_requested_chunks_have_the_same_bits(samples, kw):
    """Rays along z, one column and one cell per sample each: no sums of several updates."""
    gen = torch.Generator().manual_seed(samples)
    dims, pd = (6, 7, samples + 2), 0.1
    grid = torch.rand(*dims, 4, generator=gen) * 0.9 + 0.05
    grid[..., 3] *= 0.05
    org = pg.grid_origin(grid.shape, pd)
    i, j = (t.reshape(-1) for t in torch.meshgrid(torch.arange(6), torch.arange(7), indexing="ij"))
    o = torch.stack([org[0] + i * pd + 0.01, org[1] + j * pd - 0.01, torch.full((42,), org[2] - pd + 0.013)], 1)
    d = torch.tensor([[0.0, 0.0, 1.0]]).expand(42, 3).contiguous()
    t = torch.rand(42, 4, generator=gen)
    grads = []
    for chunk in (0, 64):
        step = pg.FusedTrainStep(grid.to(DEV), pd, samples, pd, mode="nearest", chunk_samples=chunk, **kw)
        step.step_rays(o.to(DEV), d.to(DEV), t.to(DEV))
        grads.append(step.grad.cpu())
    assert torch.equal(grads[0], grads[1])
