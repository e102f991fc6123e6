"""Roundings that the render kernels keep: a trilinear sample's blend is the reference's, bit for
bit, and a nearest ray without early stop has the gradient of one long chunk whatever chunks it
runs in. (An ulp of an opacity near 1 is 6e-4 of the beta term's gradient.)"""
import numpy as np
import pytest
import torch

import plenoxels_gb300 as pg
from oracle import torch_port as tp

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("mode", ["nearest", "trilinear"])
@pytest.mark.parametrize("lo,hi", [(0.0, 1.0), (-0.3, 1.3), (0.999, 1.0)])
def test_one_sample_has_the_reference_bits(mode, lo, hi):
    rng = np.random.default_rng(3)
    grid = torch.from_numpy(rng.uniform(lo, hi, (20, 21, 19, 4)).astype(np.float32))
    o = torch.from_numpy(rng.uniform(-0.8, 0.8, (4000, 3)).astype(np.float32))
    d = rng.normal(size=(4000, 3))
    d = torch.from_numpy((d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32))
    ref = tp.render(grid, o, d, 1, 0.05, tp.grid_min(grid.shape, 0.1), 0.1, mode)
    got = pg.render_rays(grid.to(DEV), o.to(DEV), d.to(DEV), 0.05, 1, 0.1, mode=mode)
    step = pg.FusedTrainStep(grid.to(DEV), 0.1, 1, 0.05, mode=mode)
    rgba = torch.empty(4000, 4, device=DEV)
    step.step_rays(o.to(DEV), d.to(DEV), torch.zeros(4000, 4, device=DEV), rgba_out=rgba)
    assert torch.equal(got.cpu(), ref) and torch.equal(rgba.cpu(), ref)


@pytest.mark.parametrize("samples", [129, 150, 256])
@pytest.mark.parametrize("kind", ["beta", "no clip"])
def test_long_nearest_rays_keep_their_bits(samples, kind):
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
    for chunk in (0, 256):
        step = pg.FusedTrainStep(grid.to(DEV), pd, samples, pd, mode="nearest", clip=kind == "beta",
                                 beta=5e-3 if kind == "beta" else 0.0, chunk_samples=chunk)
        step.step_rays(o.to(DEV), d.to(DEV), t.to(DEV))
        grads.append(step.grad.cpu())
    assert torch.equal(grads[0], grads[1])
