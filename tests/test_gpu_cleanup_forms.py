"""The clean-up's form with 4 bytes of scratch a cell (pgb_remove_noise), which also takes over
where the planes' scratch does not fit: against the oracle and against the planes' form."""
import numpy as np
import pytest
import torch

import plenoxels_gb300 as pg
from oracle import torch_port as tp
from plenoxels_gb300 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"

CASES = [((1, 1, 1), 3, 1.0, 0.5, 3), ((5, 9, 130), 3, 1.0, 1.5, 1), ((5, 9, 130), 3, 1.0, 1.5, 12),
         ((14, 13, 12), 7, 3.0, 9.0, 4), ((14, 13, 12), 5, 1.0, 0.25, 2), ((14, 13, 12), 3, 1.0, 1.0, 0)]


def _grid(dims, seed):
    rng = np.random.default_rng(seed)
    g = torch.from_numpy(rng.uniform(-0.2, 1.0, (*dims, 4)).astype(np.float32))
    g[..., 3][torch.from_numpy(rng.random(dims) < 0.5)] = 0.0
    g[..., 3][torch.from_numpy(rng.random(dims) < 0.1)] = -0.0
    return g


@pytest.mark.parametrize("dims,kernel,radius,threshold,repeats", CASES)
def test_small_scratch(dims, kernel, radius, threshold, repeats):
    g = _grid(dims, kernel)
    got = g.to(DEV)
    sums = torch.empty(dims, device=DEV)
    _lib.check(_lib.load().pgb_remove_noise(got.data_ptr(), _lib.dims3(dims), kernel, radius, threshold,
                                            repeats, sums.data_ptr(), _lib.stream_of(got)), "clean-up")
    assert torch.equal(got.cpu(), tp.remove_noise(g.clone(), kernel, radius, threshold, repeats))


@pytest.mark.parametrize("dims,kernel,radius,threshold,repeats", CASES)
def test_planes_that_do_not_fit(dims, kernel, radius, threshold, repeats, monkeypatch):
    g = _grid(dims, kernel).to(DEV)
    want = pg.convolve_grid_to_remove_noise(g.clone(), kernel, radius, threshold, repeats)
    empty = torch.empty

    def full(*args, **kw):
        if kw.get("dtype") is torch.uint8:
            raise torch.cuda.OutOfMemoryError("no room for the planes")
        return empty(*args, **kw)

    monkeypatch.setattr(torch, "empty", full)
    got = pg.convolve_grid_to_remove_noise(g.clone(), kernel, radius, threshold, repeats)
    monkeypatch.undo()
    assert torch.equal(got, want)
