"""Batches whose scenes need different index arithmetic, in one launch: centred ones, scenes with
an origin component of 0 or next to it, an axis of one or two cells, an extreme pitch; against
the oracle, and with coordinates that are bit for bit those of the single-scene kernels."""
import numpy as np
import pytest
import torch

from oracle import torch_port as tp
from plenoxels_gb300.batch import BatchedTrainStep, Scene

pytestmark = pytest.mark.gpu
DEV = "cuda"

CENTRED, ZERO = "centred", (0.0, 0.0, 0.0)
KINDS = {  # dims, pitch, origin
    "centred": ((20, 21, 22), 0.1, CENTRED), "zero": ((21, 20, 19), 0.1, ZERO),
    "near zero": ((20, 23, 21), 0.1, (1e-7, -0.9, -1e-30)), "slab": ((24, 2, 25), 0.1, CENTRED),
    "line": ((1, 1, 40), 0.05, CENTRED), "tiny": ((20, 21, 22), 1e-13, CENTRED),
    "tiny at zero": ((20, 21, 22), 1e-13, ZERO), "huge": ((20, 21, 22), 1e13, ZERO)}
BATCHES = [["centred", "zero", "centred"], ["zero", "zero"], ["tiny"], list(KINDS), ["tiny at zero", "centred"]]


def _scene(kind, rays, S, rng, dtype):
    dims, pd, origin = KINDS[kind]
    gmin = tp.grid_min(torch.Size([*dims, 4]), pd) if origin == CENTRED else torch.tensor(origin)
    occ = torch.from_numpy(rng.random(dims) < 0.5)
    cells = torch.from_numpy(rng.uniform(0.0, 1.0, (*dims, 4)).astype(np.float32))
    cells[..., 3] *= 0.2
    cells[~occ] = 0.0
    cells = cells.to(dtype)
    delta = float(np.float32(1.6 * max(dims) * pd / S))
    d = rng.normal(size=(rays, 3)) * np.minimum(np.array(dims) / 10.0, 1.0)
    d = torch.from_numpy((d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32))
    jitter = rng.uniform(-0.3, 0.3, (rays, 3)) * np.array(dims) * pd
    o = gmin + torch.tensor(dims) * pd / 2 + torch.from_numpy(jitter.astype(np.float32)) - 0.5 * S * delta * d
    target = torch.from_numpy(rng.random((rays, 4)).astype(np.float32))
    own = None if origin == CENTRED else tuple(gmin.tolist())
    return dict(cells=cells, occ=occ, gmin=gmin, own=own, pd=pd, delta=delta, S=S, o=o.contiguous(), d=d, t=target)


@pytest.mark.parametrize("kinds", BATCHES, ids=lambda k: "+".join(k))
@pytest.mark.parametrize("mode", ["nearest", "trilinear"])
@pytest.mark.parametrize("tile", [(1, 256, 1), (1, 128, 0), (2, 256, 0), (8, 128, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_mixed_scenes_match_the_oracle(kinds, mode, tile, dtype):
    rng = np.random.default_rng(len(kinds))
    problem = [_scene(k, 40 + 25 * i, 90 + 50 * (i % 3), rng, dtype) for i, k in enumerate(kinds)]
    R = sum(p["o"].shape[0] for p in problem)
    step = BatchedTrainStep([Scene(p["cells"].to(DEV), p["occ"].to(DEV), p["pd"], p["S"], p["delta"], p["own"])
                             for p in problem], R, mode=mode, term_threshold=0.0, tiles=tile)
    step.rgba = torch.empty(R, 4, device=DEV)
    own = torch.cat([torch.full((p["o"].shape[0],), i, dtype=torch.int32) for i, p in enumerate(problem)])
    mix = torch.from_numpy(rng.permutation(R))   # rays of all scenes in any order
    step.set_rays(*(torch.cat([p[k] for p in problem])[mix].to(DEV) for k in "odt"), own[mix].to(DEV))
    for _ in range(2):   # the second step finds the counters of the first
        step.rgba.zero_()
        loss = step.step()
        want, total = [], 0.0
        for p, scene in zip(problem, step.scenes):
            g = p["cells"].float().clone().requires_grad_(True)
            px = tp.render(g, p["o"], p["d"], p["S"], p["delta"], p["gmin"], p["pd"], mode)
            sq = ((px - p["t"]) ** 2).sum()
            (sq / (4 * R)).backward()
            want.append(px.detach())
            total += float(sq.detach()) / (4 * R)
            ref = g.grad * p["occ"].unsqueeze(-1)
            assert float((scene.grad.cpu() - ref).abs().max()) <= 1e-4 * float(ref.abs().max())
        np.testing.assert_allclose(step.rgba.cpu().numpy(), torch.cat(want)[mix].numpy(), rtol=1e-5, atol=2e-6)
        np.testing.assert_allclose(float(loss), total, rtol=1e-5)
