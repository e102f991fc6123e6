"""The quick index arithmetic and the cut of a ray to the samples that can be in bounds,
where they can go wrong: quotients by the cell pitch at awkward pitches, rays along and
beside the grid's faces, cells at the clamp's edges and NaN cells, grids outside the quick
range. Against fp32 numpy (coordinates, bit for bit) and the oracle."""
from fractions import Fraction

import numpy as np
import pytest
import torch

import plenoxels_gb300 as pg
from plenoxels_gb300 import _lib
from plenoxels_gb300.render import _rays_desc
from oracle import torch_port as tp

DEV = "cuda"


def _round32(x: Fraction) -> np.float32:
    """The fp32 number nearest to x, ties to even (normal range)."""
    if x == 0:
        return np.float32(0)
    n, d = abs(x).numerator, abs(x).denominator
    e = n.bit_length() - d.bit_length()
    e -= Fraction(n, d) < Fraction(2) ** e
    q = abs(x) / Fraction(2) ** (e - 23)
    m = q.numerator // q.denominator
    r = q - m
    m += r > Fraction(1, 2) or (r == Fraction(1, 2) and m % 2 == 1)
    return np.float32((1 if x > 0 else -1) * float(Fraction(m) * Fraction(2) ** (e - 23)))


@pytest.mark.parametrize("pd", [3.0 / 256, 3.0 / 7, 0.1, 1.0, np.float32(2) - np.float32(2 ** -23),
                                np.float32(1) + np.float32(2 ** -23), 1e-9, 3.3e9])
def test_reciprocal_with_two_corrections_is_the_rounded_quotient(pd):
    """The kernels' division by the pitch (product with the rounded reciprocal, then twice
    q += (x - q pd) y, fused) in exact arithmetic, against the IEEE quotient."""
    pd = np.float32(pd)
    y = np.float32(1) / pd
    rng = np.random.default_rng(3)
    xs = (rng.uniform(-8, 8, 1500) * float(pd) * 2.0 ** rng.integers(-20, 9, 1500)).astype(np.float32)
    F = lambda v: Fraction(float(v))  # noqa: E731
    for x in np.concatenate([xs, [np.float32(0), pd, -pd]]).astype(np.float32):
        q = _round32(F(x) * F(y))
        for _ in range(2):
            r = _round32(F(x) - F(q) * F(pd))
            q = _round32(F(r) * F(y) + F(q))
        assert q == x / pd


def _render_masked(g, o, d, S, delta, gmin, pd, mode):
    """tp.render with the samples outside the grid replaced by 0. (The reference multiplies
    by the mask, which keeps a NaN that an outside sample's wrapped indices fetch; the fused
    kernels read no cell for such a sample.)"""
    n = tp.normalize(tp.sample_positions(o, d, S, delta), gmin, pd)
    look = tp.nearest_lookup if mode == "nearest" else tp.trilinear_lookup
    vals, mask, _ = look(n, g.clip(0, 1))
    vals = torch.where(mask.unsqueeze(-1), vals, torch.zeros(()))
    return tp.composite(vals.reshape(1, o.shape[0], S, 4)).reshape(-1, 4)


def _special_rays(dims, pd, rng, n=400):
    """Origins and directions [n,3]: through the box, along its axes (two zero components),
    inside its faces and just outside them, starting inside, missing it, pointing away."""
    half = np.array(dims) * pd / 2
    o = rng.normal(size=(n, 3)) * 2.0
    d = rng.normal(size=(n, 3))
    kind = np.arange(n) % 6
    for i in range(n):
        ax = int(rng.integers(3))
        if kind[i] == 1:
            d[i] = 0.0
            d[i, ax] = rng.choice([-1.0, 1.0])
            o[i] = rng.uniform(-1, 1, 3) * half
            o[i, ax] = -d[i, ax] * (half[ax] + 1.0)
        elif kind[i] == 2:  # along a face, within a few ulp of the bounds
            lo = (1 - np.ceil(np.array(dims) / 2)) * pd
            edge = [lo[ax], lo[ax] - 0.5 * pd, lo[ax] + dims[ax] * pd, lo[ax] + (dims[ax] - 0.5) * pd]
            d[i, ax] = 0.0
            o[i] = -3.0 * d[i] / np.linalg.norm(d[i])
            o[i, ax] = edge[int(rng.integers(4))] * (1 + rng.integers(-2, 3) * 2.0 ** -24)
        elif kind[i] == 3:
            o[i] = rng.uniform(-0.9, 0.9, 3) * half
        elif kind[i] == 4:
            o[i] = rng.normal(size=3) * 5 + 4
        else:
            o[i] = -2.5 * d[i] / np.linalg.norm(d[i]) + rng.uniform(-0.5, 0.5, 3)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return torch.from_numpy(o.astype(np.float32)), torch.from_numpy(d.astype(np.float32))


@pytest.mark.gpu
@pytest.mark.parametrize("dims,pd", [((7, 33, 20), 0.1), ((64, 50, 3), 3.0 / 64), ((5, 1, 9), 0.3),
                                     ((40, 40, 40), 1e-9), ((300, 2, 90), 1.7)])
def test_coordinates_are_the_rounded_ones(dims, pd):
    o, d = _special_rays(dims, pd, np.random.default_rng(5))
    S, delta = 70, 0.09
    g = torch.zeros(*dims, 4, device=DEV)
    org = pg.grid_origin(g.shape, pd)
    out = torch.empty(o.shape[0], S, 3, device=DEV)
    gd = _lib.make_grid(g, org, pd, _lib.PGB_TRILINEAR, True)
    od, dd = o.to(DEV), d.to(DEV)
    rd = _rays_desc(od, dd, o.shape[0], S, delta, False, 0, 0.0)
    _lib.check(_lib.load().pgb_render_sample_coords(gd, rd, out.data_ptr(), 0), "coords")
    ref = tp.normalize(tp.sample_positions(o, d, S, delta), torch.tensor(org), pd)
    np.testing.assert_array_equal(out.cpu().numpy().reshape(-1, 3), ref.numpy())


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["nearest", "trilinear"])
@pytest.mark.parametrize("dims,S,delta,thr", [((7, 33, 20), 70, 0.09, 0.0), ((64, 50, 40), 300, 0.02, 0.0),
                                              ((64, 50, 40), 300, 0.02, 1e-3), ((5, 1, 9), 33, 0.2, 0.0),
                                              ((20, 20, 20), 1, 2.0, 0.0), ((20, 20, 20), 40, -0.1, 0.0)])
def test_special_rays_match_the_oracle(mode, dims, S, delta, thr):
    rng = np.random.default_rng(11)
    pd = 2.0 / max(dims)
    o, d = _special_rays(dims, pd, rng)
    grid = torch.from_numpy(rng.uniform(-0.1, 1.1, (*dims, 4)).astype(np.float32))
    grid[..., 3] *= 0.1
    target = torch.from_numpy(rng.random((o.shape[0], 4)).astype(np.float32))
    gmin = tp.grid_min(grid.shape, pd)
    g = grid.clone().requires_grad_(True)
    px = tp.render(g, o, d, S, delta, gmin, pd, mode)
    loss = torch.nn.functional.mse_loss(px, target)
    loss.backward()
    step = pg.FusedTrainStep(grid.to(DEV), pd, S, delta, mode=mode, term_threshold=thr)
    rgba = torch.empty(o.shape[0], 4, device=DEV)
    got = step.step_rays(o.to(DEV), d.to(DEV), target.to(DEV), rgba_out=rgba)
    # a ray that stops at transmittance thr leaves out at most thr of every channel
    np.testing.assert_allclose(rgba.cpu().numpy(), px.detach().numpy(), rtol=1e-5, atol=2e-6 + thr)
    np.testing.assert_allclose(float(got), float(loss.detach()), rtol=1e-5 + thr)
    if thr == 0.0:
        scale = g.grad.abs().max()
        assert (step.grad.cpu() - g.grad).abs().max() <= 1e-4 * scale
        fwd = pg.render_rays(grid.to(DEV), o.to(DEV), d.to(DEV), delta, S, pd, mode=mode)
        assert torch.equal(fwd, rgba)
        # the beta term counts the samples outside the grid too
        _, vals = tp.render_samples(grid, o, d, S, delta, gmin, pd, mode)
        beta = tp.beta_loss(vals[..., 3].double())
        step = pg.FusedTrainStep(grid.to(DEV), pd, S, delta, mode=mode, beta=5e-3)
        step.step_rays(o.to(DEV), d.to(DEV), target.to(DEV))
        np.testing.assert_allclose(float(step.losses[1]), 5e-3 * float(beta), rtol=1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["nearest", "trilinear"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_clamp_edges_and_nan_cells(mode, dtype):
    """Values at the clamp's edges pass the gradient where the reference's clamp does (0,
    -0 and 1 inside), infinities clamp, NaN cells make their rays NaN and no others."""
    rng = np.random.default_rng(2)
    dims, pd, S, delta = (20, 21, 22), 0.1, 64, 0.05
    grid = torch.from_numpy(rng.uniform(0.0, 0.2, (*dims, 4)).astype(np.float32)).to(dtype)
    edge = torch.tensor([0.0, -0.0, 1.0, -1e-30, 1.0078125, float("inf"), -float("inf")]).to(dtype)
    pick = torch.from_numpy(rng.integers(0, 60, grid.shape))
    for i, v in enumerate(edge):
        grid[..., :3][pick[..., :3] == i] = v
    grid[..., 3][pick[..., 3] < 2] = 0.0
    grid[..., 3][pick[..., 3] == 1] = -0.0
    grid[3, 4, 5, 1] = float("nan")
    grid[12, 10, 11, 3] = float("nan")
    o, d = _special_rays(dims, pd, rng, 300)
    target = torch.from_numpy(rng.random((300, 4)).astype(np.float32))
    g = grid.float().clone().requires_grad_(True)
    gmin = tp.grid_min(grid.shape, pd)
    px = _render_masked(g, o, d, S, delta, gmin, pd, mode)
    bad = torch.isnan(px).any(1)
    assert 0 < int(bad.sum()) < 300
    step = pg.FusedTrainStep(grid.to(DEV), pd, S, delta, mode=mode)
    rgba = torch.empty(300, 4, device=DEV)
    step.step_rays(o.to(DEV), d.to(DEV), target.to(DEV), rgba_out=rgba)
    np.testing.assert_allclose(rgba.cpu().numpy(), px.detach().numpy(), rtol=1e-5, atol=2e-6)
    fwd = pg.render_rays(grid.to(DEV), o.to(DEV), d.to(DEV), delta, S, pd, mode=mode)
    np.testing.assert_array_equal(fwd.cpu().numpy(), rgba.cpu().numpy())
    # the gradient of the rays that meet no NaN
    keep = ~bad
    torch.nn.functional.mse_loss(_render_masked(g, o[keep], d[keep], S, delta, gmin, pd, mode),
                                 target[keep]).backward()
    step.step_rays(o[keep].to(DEV), d[keep].to(DEV), target[keep].to(DEV))
    assert (step.grad.cpu() - g.grad).abs().max() <= 1e-4 * g.grad.abs().max()
    zero = (grid.float() == 0) & (g.grad != 0)
    assert int(zero.sum()) > 0 and bool((step.grad.cpu()[zero] != 0).all())
