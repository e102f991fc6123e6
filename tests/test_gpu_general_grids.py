"""fp32 and BF16 grids outside the quick index arithmetic's range (an origin component near 0,
a tiny pitch): chunk sizes and the threshold on the transmittance as for any other grid."""
import numpy as np
import pytest
import torch

import plenoxels_gb300 as pg
from oracle import torch_port as tp

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("origin", ["centred", "zero"])
@pytest.mark.parametrize("mode", ["nearest", "trilinear"])
@pytest.mark.parametrize("transmittance", ["product", "logsum"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("chunk", [0, 32, 64, 128, 256, 512])
def test_threshold_is_looked_at_after_every_chunk(origin, mode, transmittance, dtype, chunk):
    """Rays along z through cells of one opacity: the first chunk that ends below the threshold
    is the ray's last."""
    a, S, thr, pd = 0.015625, 600, 0.7, 0.25
    grid = torch.full((4, 5, 640, 4), a, dtype=dtype, device=DEV)
    org = pg.grid_origin(grid.shape, pd) if origin == "centred" else (0.0, 0.0, 0.0)
    o = torch.tensor([[org[0] + 1.05 * pd, org[1] + 2.1 * pd, org[2] + 0.05 * pd]], device=DEV).repeat(70, 1)
    d = torch.tensor([[0.0, 0.0, 1.0]], device=DEV).repeat(70, 1)
    c = chunk or (64 if mode == "nearest" else 32)
    n = next(k for k in range(c, S + c, c) if (1 - a) ** k < thr)
    want = 1 - (1 - a) ** min(n, S)
    kw = dict(mode=mode, transmittance=transmittance, chunk_samples=chunk, term_threshold=thr)
    step = pg.FusedTrainStep(grid, pd, S, pd, grid_min=org, **kw)
    rgba = torch.empty(70, 4, device=DEV)
    step.step_rays(o, d, torch.zeros(70, 4, device=DEV), rgba_out=rgba)
    fwd = pg.render_rays(grid, o, d, pd, S, pd, org, **kw)
    # a product or sum of at most 600 fp32 factors, rounded once each
    np.testing.assert_allclose(rgba[:, 3].cpu().numpy(), want, atol=600 * 2.0 ** -24)
    np.testing.assert_allclose(fwd[:, 3].cpu().numpy(), want, atol=600 * 2.0 ** -24)
    hit = (step.grad[..., 3] != 0).any(0).any(0).nonzero()
    # sample k lies 0.05 beyond cell k: trilinear lookup reads the next cell too
    assert int(hit.max()) == min(n, S) + (1 if mode == "trilinear" else 0)


@pytest.mark.parametrize("origin,dims,pd", [("zero", (30, 33, 28), 0.1), ("centred", (30, 2, 28), 0.1),
                                            ("centred", (30, 33, 28), 1e-13)])
@pytest.mark.parametrize("mode", ["nearest", "trilinear"])
@pytest.mark.parametrize("chunk", [0, 32, 64, 128, 256, 512])
@pytest.mark.parametrize("kw", [{}, dict(beta=5e-3), dict(clip=False)], ids=["", "beta", "no clip"])
def test_every_chunk_size_matches_the_oracle(origin, dims, pd, mode, chunk, kw):
    rng = np.random.default_rng(chunk)
    S, R = 300, 200
    gmin = tp.grid_min(torch.Size([*dims, 4]), pd) if origin == "centred" else torch.zeros(3)
    delta = 1.5 * 30 * pd / S
    grid = torch.from_numpy(rng.uniform(0.0, 1.0, (*dims, 4)).astype(np.float32))
    grid[..., 3] = 0.02 + 0.1 * grid[..., 3]
    mid = gmin + torch.tensor(dims) * pd / 2
    d = rng.normal(size=(R, 3)) * [1.0, 0.02 if dims[1] == 2 else 1.0, 1.0]
    d = torch.from_numpy((d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32))
    o = (mid + torch.from_numpy((rng.uniform(-0.2, 0.2, (R, 3)) * pd * np.array(dims)).astype(np.float32))
         - 0.5 * S * delta * d)
    target = torch.from_numpy(rng.random((R, 4)).astype(np.float32))
    g = grid.clone().requires_grad_(True)
    px, vals = tp.render_samples(g, o, d, S, delta, gmin, pd, mode, clip=kw.get("clip", True))
    loss = torch.nn.functional.mse_loss(px, target)
    if "beta" in kw:
        loss = loss + 5e-3 * tp.beta_loss(vals[..., 3])
    loss.backward()
    step = pg.FusedTrainStep(grid.to(DEV), pd, S, delta, mode=mode, chunk_samples=chunk,
                             grid_min=tuple(gmin.tolist()), **kw)
    rgba = torch.empty(R, 4, device=DEV)
    step.step_rays(o.to(DEV), d.to(DEV), target.to(DEV), rgba_out=rgba)
    np.testing.assert_allclose(rgba.cpu().numpy(), px.detach().numpy(), rtol=1e-5, atol=2e-6)
    assert (step.grad.cpu() - g.grad).abs().max() <= 1e-4 * g.grad.abs().max()
    fwd = pg.render_rays(grid.to(DEV), o.to(DEV), d.to(DEV), delta, S, pd, tuple(gmin.tolist()), mode=mode,
                         chunk_samples=chunk, clip=kw.get("clip", True))
    np.testing.assert_allclose(fwd.cpu().numpy(), px.detach().numpy(), rtol=1e-5, atol=2e-6)
