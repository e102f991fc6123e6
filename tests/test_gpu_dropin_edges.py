"""Drop-in operators at the edges of their vector forms: odd counts, tables that are not
16-byte aligned, indices far outside the grid. Bit for bit against
the oracle's restatement of the reference (on the CPU)."""
import numpy as np
import pytest
import torch

import plenoxels_gb300 as pg
from oracle import torch_port as tp

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _offset(t, by):
    """t on the GPU in storage that starts `by` elements into an allocation."""
    base = torch.empty(t.numel() + by, dtype=t.dtype, device=DEV)
    view = base[by:].view(t.shape)
    view.copy_(t)
    return view


@pytest.mark.parametrize("count", [1, 2, 3, 5, 31, 257, 1000])
@pytest.mark.parametrize("by", [0, 1])
def test_lookup_chain(count, by):
    rng = np.random.default_rng(count)
    dims = (9, 7, 12)
    grid = torch.from_numpy(rng.uniform(-0.5, 1.5, (*dims, 4)).astype(np.float32))
    n = torch.from_numpy((rng.uniform(-1.2, 2.2, (count, 3)) * np.array(dims)).astype(np.float32))
    n[::7] = n[::7].round()
    nd = _offset(n, by)
    corners = tp.corner_indices(n)
    got = pg.get_grid_points_indices(nd)
    assert torch.equal(got.cpu(), corners)
    wrapped = tp.wrap_(corners.clone().view(-1, 3), dims).view(-1, 8, 3)
    idx = _offset(corners, by)
    pg.fix_out_of_bounds(idx.view(-1, 3), grid.to(DEV))
    assert torch.equal(idx.cpu(), wrapped)
    ref = tp.trilinear_blend(n, wrapped, grid.clip(0, 1))
    g = grid.to(DEV).requires_grad_(True)
    vals = pg.trilinear_interpolation(nd, idx, g, clip=True)
    assert torch.equal(vals.detach().cpu(), ref)
    d = torch.from_numpy(rng.normal(size=(count, 4)).astype(np.float32))
    vals.backward(d.to(DEV))
    gr = grid.clone().requires_grad_(True)
    tp.trilinear_blend(n, wrapped, gr.clip(0, 1)).backward(d)
    # the same products added in another order: at most a few hundred terms of size 1
    assert (g.grad.cpu() - gr.grad).abs().max() <= 1e-4 * gr.grad.abs().max()
    near, mask = pg.get_nearest_voxels(nd, g.detach())
    ref_v, ref_m, _ = tp.nearest_lookup(n, grid)
    assert torch.equal(near.cpu(), ref_v) and torch.equal(mask.cpu(), ref_m)


@pytest.mark.parametrize("count", [1, 3, 4, 5, 1023])
@pytest.mark.parametrize("by", [0, 1, 2])
def test_normalisation_of_any_alignment(count, by):
    rng = np.random.default_rng(count + by)
    table = torch.from_numpy(rng.normal(size=(count, 3)).astype(np.float32))
    samples = torch.from_numpy(rng.normal(size=(2 * count + 1, 3)).astype(np.float32))
    got = pg.normalize_samples_for_indecies(_offset(table, by), _offset(samples, by), 0.3)
    assert torch.equal(got.cpu(), (samples - table.min(0)[0]) / 0.3)


def test_wrapping_of_distant_indices():
    vals = torch.tensor([0, 6, 7, -1, -7, -8, 13, 14, 15, 10 ** 12, -10 ** 12, 2 ** 31, -2 ** 31, 2 ** 62,
                         -2 ** 62, 5], dtype=torch.int64)
    idx = torch.stack([vals, vals.flip(0), vals.roll(3)], 1)
    shape = (7, 1, 300, 4)
    ref = tp.wrap_(idx.clone(), shape)
    got = idx.to(DEV)
    pg.fix_out_of_bounds(got, torch.empty(shape, device=DEV))
    assert torch.equal(got.cpu(), ref)
