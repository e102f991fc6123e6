"""render_rays under torch's tracing, transforms, forward mode and inference mode: a call
without a gradient leaves its autograd Function out, and behaves as with it everywhere."""
import pytest
import torch

import plenoxels_gb300 as pg
from plenoxels_gb300.inference import render_camera_images
from plenoxels_gb300.render import _wants_autograd

DEV = "cuda"


def test_which_calls_take_the_function():
    x = torch.ones(3)
    leaf = torch.ones(3, requires_grad=True)
    assert not _wants_autograd(x) and _wants_autograd(x, leaf)
    with torch.no_grad():
        assert not _wants_autograd(leaf)
    with torch.inference_mode():
        assert not _wants_autograd(leaf)
    with torch.autograd.forward_ad.dual_level():
        assert _wants_autograd(x)
    seen = []
    torch.func.vmap(lambda v: seen.append(_wants_autograd(v)) or v)(x)
    with torch.no_grad():
        torch.jit.trace(lambda v: seen.append(_wants_autograd(v)) or v + 1, x, check_trace=False)
    assert seen == [True, True] and not _wants_autograd(x)


def _scene():
    gen = torch.Generator(device=DEV).manual_seed(8)
    grid = torch.rand(20, 21, 22, 4, generator=gen, device=DEV)
    grid[..., 3] *= 0.1
    o = torch.rand(50, 3, generator=gen, device=DEV) * 0.4 + torch.tensor([0.0, 0.0, 2.5], device=DEV)
    d = torch.nn.functional.normalize(torch.randn(50, 3, generator=gen, device=DEV) * 0.2
                                      - torch.tensor([0.0, 0.0, 1.0], device=DEV), dim=1)
    return grid, o, d


def _render(grid, o, d):
    return pg.render_rays(grid, o, d, 0.04, 100, 0.1)


@pytest.mark.gpu
def test_traced_calls_render_their_own_rays():
    grid, o, d = _scene()
    with torch.no_grad():
        traced = torch.jit.trace(_render, (grid, o, d), check_trace=False)
        torch.empty(50, 4, device=DEV).fill_(7.0)   # what a fresh buffer may hold
        other = (grid.flip(0).contiguous(), o + 0.05, d)
        assert torch.equal(traced(*other), _render(*other))


@pytest.mark.gpu
def test_inference_mode_renders_the_same():
    grid, o, d = _scene()
    with torch.inference_mode():
        got = _render(grid, o, d)
    assert torch.equal(got, _render(grid, o, d))
    assert torch.equal(got, _render(grid.requires_grad_(True), o, d))


@pytest.mark.gpu
def test_transforms_and_forward_mode_are_refused():
    grid, o, d = _scene()
    with torch.no_grad(), pytest.raises(RuntimeError):
        torch.func.vmap(lambda v: _render(grid, v, d))(torch.stack([o, o]))
    T = torch.eye(4, device=DEV)[None].clone()
    T[0, 2, 3] = 2.5
    with torch.autograd.forward_ad.dual_level():
        for run, x in ((lambda g: _render(g, o, d), grid), (lambda v: _render(grid, v, d), o),
                       (lambda c: render_camera_images(grid, c, 8, 8, 0.7, 0.1, 0.04, 100, 0.1), T)):
            dual = torch.autograd.forward_ad.make_dual(x, torch.ones_like(x))
            with torch.no_grad(), pytest.raises(RuntimeError):
                run(dual)
