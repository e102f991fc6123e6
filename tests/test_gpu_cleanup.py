"""The stray-cell clean-up's repeats at small and ragged grids, against the oracle."""
import numpy as np
import pytest
import torch

import plenoxels_gb300 as pg
from oracle import torch_port as tp

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dims,kernel,radius,threshold,repeats", [
    ((1, 1, 1), 3, 1.0, 0.5, 3), ((5, 9, 130), 3, 1.0, 1.5, 1), ((5, 9, 130), 3, 1.0, 1.5, 12),
    ((14, 13, 12), 7, 3.0, 9.0, 4), ((14, 13, 12), 5, 1.0, 0.0, 2), ((14, 13, 12), 3, 1.0, 1.0, 0),
    ((14, 13, 12), 5, 2.2, -0.3, 5)])
def test_cleanup(dims, kernel, radius, threshold, repeats):
    rng = np.random.default_rng(kernel)
    g = torch.from_numpy(rng.uniform(-0.2, 1.0, (*dims, 4)).astype(np.float32))
    g[..., 3][torch.from_numpy(rng.random(dims) < 0.5)] = 0.0
    g[..., 3][torch.from_numpy(rng.random(dims) < 0.1)] = -0.0
    ref = tp.remove_noise(g.clone(), kernel, radius, threshold, repeats)
    got = pg.convolve_grid_to_remove_noise(g.to(DEV), kernel, radius, threshold, repeats).cpu()
    # a cell whose sum lies within the rounding of a threshold may fall either way
    assert float((got != ref).any(-1).float().mean()) <= (0.0 if threshold > 0 else 0.02)
