"""The views of the fused kernels' sample coordinates at positions that overflow: the IEEE
quotient's infinities and NaN."""
import numpy as np
import pytest
import torch

import plenoxels_gb300 as pg
from oracle import torch_port as tp
from plenoxels_gb300 import _lib
from plenoxels_gb300.render import _rays_desc

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("pd", [0.1, 1e-9, 3.0])
def test_coordinates_that_are_not_finite(pd):
    inf = float("inf")
    o = torch.tensor([[inf, 0.0, 1.0], [-inf, 1.0, 0.5], [3e38, -3e38, 0.2], [0.0, float("nan"), 1e30],
                      [0.1, 0.2, 0.3], [0.0, 0.0, 0.0]])
    d = torch.tensor([[0.0, 0.0, -1.0], [0.6, 0.8, 0.0], [1e38, 0.0, 0.0], [0.0, 1.0, 0.0],
                      [inf, 0.0, 0.0], [0.0, -inf, 0.0]])
    grid = torch.zeros(20, 21, 22, 4, device=DEV)
    org = pg.grid_origin(grid.shape, pd)
    out = torch.empty(6, 40, 3, device=DEV)
    od, dd = o.to(DEV), d.to(DEV)
    gd = _lib.make_grid(grid, org, pd, _lib.PGB_NEAREST, True)
    rd = _rays_desc(od, dd, 6, 40, 0.09, False, 0, 0.0)
    _lib.check(_lib.load().pgb_render_sample_coords(gd, rd, out.data_ptr(), 0), "coords")
    ref = tp.normalize(tp.sample_positions(o, d, 40, 0.09), torch.tensor(org), pd)
    np.testing.assert_array_equal(out.cpu().numpy().reshape(-1, 3), ref.numpy())
