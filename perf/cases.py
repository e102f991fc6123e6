"""The work that users of the package have it do, as measurable cases.

Scenes are those of the repository's benchmark and tests: a dense [X,Y,Z,4] grid of Gaussian
blobs (RGB = sigmoid of normals) in the box [-1.5, 1.5]^3, seen by look-at pinhole cameras at
radius 4 on the upper hemisphere (field of view 0.691 rad, rays from near 2 to far 6). Every
case goes through the package's public entry points and returns what they compute, whole.

Kinds of case (``kind``):

  render         render_rays without gradients: a batch of rays to pixels
  autograd       render_rays with its backward through torch autograd (dense grid gradient)
  step_rays      FusedTrainStep on explicit rays: loss and dense gradient
  step_cameras   FusedTrainStep on rays generated from cameras and their images
  trainer        Trainer.step_rays: render, beta and TV loss, backward, Adam, |grad| sum
  growing        the same with progressive growing (the pooled grid of a receptive field)
  batched        BatchedTrainStep over many sparse scenes
  dropin         the training step composed from the drop-in functions of the reference
  images         inference.render_camera_images: whole pictures
  clean          convolve_grid_to_remove_noise on a copy of the grid
"""
from __future__ import annotations

import math

import numpy as np
import torch

import plenoxels_gb300 as pg
from plenoxels_gb300.batch import BatchedTrainStep, Scene
from plenoxels_gb300.inference import render_camera_images

DEV = "cuda"
FOV = 0.691
NEAR, FAR = 2.0, 6.0
STRAT_SEED = 7
ADAM = dict(lr=0.0025, betas=(0.9, 0.999), eps=1e-8)
MOMENT_STEPS = 200   # optimiser steps the trainer cases have behind them
BETA_EPS = 1e-4
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}


def listed():
    return [
        # a probe of a few rays through a small grid, as an interactive viewer or a test
        # asks for: launch latency and the host path
        dict(name="render_probe", kind="render", x=64, y=64, z=64, rays=256, samples=128,
             mode="trilinear", dtype="f32", alpha="opaque", background=False),
        # the smallest training configuration: 64^3, one 64x64 view's rays, nearest lookup
        dict(name="step_small_nearest", kind="step_rays", x=64, y=64, z=64, rays=4096, samples=128,
             mode="nearest", dtype="f32", alpha="opaque", transmittance="product", zeroing="fill"),
        # the benchmark's training step: 8192 rays x 256 from 100 cameras, trilinear
        dict(name="step_cameras", kind="step_cameras", x=256, y=256, z=256, rays=8192, samples=256,
             mode="trilinear", dtype="f32", alpha="opaque", cameras=100, image=400,
             zeroing="marked"),
        # the precision form: 512^3 BF16 cells, log-sum transmittance, the largest step
        dict(name="step_precision", kind="step_rays", x=512, y=512, z=512, rays=65536, samples=512,
             mode="trilinear", dtype="bf16", alpha="opaque", transmittance="logsum",
             zeroing="marked"),
        # a user's own training loop over render_rays: torch loss and autograd, a ragged
        # grid that is half transparent, a white background
        dict(name="autograd_ragged", kind="autograd", x=150, y=201, z=173, rays=5003, samples=100,
             mode="trilinear", alpha="soft", background=True),
        # the whole training step at the reference's own sizes (75 rays for each of 100
        # cameras, 600 samples, nearest lookup) with its TV and beta terms
        dict(name="trainer_full", kind="trainer", x=256, y=256, z=256, rays=7500, samples=600,
             mode="nearest", tv=1e-5, beta=5e-3),
        # the same loop without the two regularisers (the reference's hard-coded run)
        dict(name="trainer_plain", kind="trainer", x=192, y=192, z=192, rays=7500, samples=600,
             mode="nearest", tv=0.0, beta=0.0),
        # coarse-to-fine training: half way down the schedule of receptive fields
        dict(name="trainer_growing", kind="growing", x=256, y=256, z=256, rays=7500, samples=600,
             mode="nearest", tv=1e-5, beta=0.0, field=21),
        # sparse scenes trained together, each with its own number of rays
        dict(name="batched_scenes", kind="batched", scenes=16, sides="32,64,128,256", samples=512,
             min_rays=1000, max_rays=64000, dtype="bf16", mode="trilinear"),
        # the reference's training step with its imports swapped for this package's
        # functions, nearest lookup (what its driver trains with)
        dict(name="dropin_nearest", kind="dropin", x=256, y=256, z=256, cameras=100, per_camera=82,
             samples=256, image=200, mode="nearest"),
        # the same composed from the trilinear functions
        dict(name="dropin_trilinear", kind="dropin", x=128, y=128, z=128, cameras=40, per_camera=75,
             samples=256, image=200, mode="trilinear"),
        # pictures of a trained grid for comparison with photographs
        dict(name="images", kind="images", x=256, y=256, z=256, cameras=3, image=400, samples=256,
             mode="trilinear", alpha="opaque"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "autograd", "step_rays", "step_cameras", "trainer", "growing",
                       "batched", "dropin", "images", "clean"])
    mode = rng.choice(["nearest", "trilinear"])

    def dims(lo, hi):
        s = _log_int(rng, lo, hi)
        if rng.random() < 0.5:
            return dict(x=s, y=s, z=s)
        return {a: max(lo, min(hi, int(s * rng.uniform(0.7, 1.3)))) for a in "xyz"}

    alpha = rng.choice(["opaque", "soft"])
    if kind == "render":
        return dict(kind=kind, **dims(32, 300), rays=_log_int(rng, 1, 400_000),
                    samples=_log_int(rng, 16, 600), mode=mode, dtype=rng.choice(["f32", "bf16"]),
                    alpha=alpha, background=rng.random() < 0.5)
    if kind == "autograd":
        return dict(kind=kind, **dims(32, 256), rays=_log_int(rng, 64, 16384),
                    samples=_log_int(rng, 32, 600), mode=mode, alpha=alpha,
                    background=rng.random() < 0.5)
    if kind == "step_rays":
        return dict(kind=kind, **dims(32, 400), rays=_log_int(rng, 256, 65536),
                    samples=_log_int(rng, 32, 600), mode=mode, dtype=rng.choice(["f32", "bf16"]),
                    alpha=alpha, transmittance=rng.choice(["product", "logsum"]),
                    zeroing=rng.choice(["fill", "marked"]))
    if kind == "step_cameras":
        return dict(kind=kind, **dims(48, 320), rays=_log_int(rng, 512, 32768),
                    samples=_log_int(rng, 64, 512), mode=mode, dtype=rng.choice(["f32", "bf16"]),
                    alpha=alpha, cameras=rng.randint(1, 100), image=rng.choice([64, 201, 400]),
                    zeroing=rng.choice(["fill", "marked"]))
    if kind == "trainer":
        return dict(kind=kind, **dims(64, 256), rays=_log_int(rng, 1024, 12800),
                    samples=_log_int(rng, 64, 600), mode=mode, tv=rng.choice([0.0, 1e-5]),
                    beta=rng.choice([0.0, 5e-3]))
    if kind == "growing":
        return dict(kind=kind, **dims(96, 256), rays=_log_int(rng, 1024, 12800),
                    samples=_log_int(rng, 64, 600), mode=mode, tv=rng.choice([0.0, 1e-5]),
                    beta=0.0, field=rng.randrange(3, 94, 2))
    if kind == "batched":
        return dict(kind=kind, scenes=rng.randint(2, 16), sides=rng.choice(["32,64", "64,128,256", "50,75,130"]),
                    samples=rng.choice([128, 300, 512]), min_rays=500, max_rays=rng.choice([4000, 32000]),
                    dtype=rng.choice(["f32", "bf16"]), mode=mode)
    if kind == "dropin":
        return dict(kind=kind, **dims(32, 192), cameras=rng.randint(1, 60), per_camera=rng.randint(20, 90),
                    samples=_log_int(rng, 32, 256), image=rng.choice([64, 150]), mode=mode)
    if kind == "images":
        return dict(kind=kind, **dims(48, 256), cameras=rng.randint(1, 4), image=_log_int(rng, 40, 400),
                    samples=_log_int(rng, 48, 400), mode=mode, alpha=alpha)
    return dict(kind=kind, **dims(32, 256), kernel=rng.choice([3, 3, 5]), threshold=rng.choice([0.5, 1.0, 2.0]))


# ------------------------------------------------------------------------------- inputs
def _pd(case):
    return 3.0 / max(case["x"], case["y"], case["z"])


def _axis(side, pd):
    return (torch.arange(side, device=DEV, dtype=torch.float32) - math.ceil(side / 2) + 1) * pd


def _blobs(dims, pd, count, gen, lo, hi, width=0.3):
    """Sum of Gaussian blobs with centres in [-1,1]^3 and amplitudes in [lo,hi]."""
    centres = torch.rand(count, 3, generator=gen, device=DEV) * 2 - 1
    amps = lo + (hi - lo) * torch.rand(count, generator=gen, device=DEV)
    axes = [_axis(s, pd) for s in dims]
    e = [torch.exp(-(axes[k][None] - centres[:, k, None]) ** 2 / (2 * width ** 2)) for k in range(3)]
    dens = torch.zeros(*dims, device=DEV)
    for i in range(count):
        dens += (amps[i] * e[0][i])[:, None, None] * e[1][i][None, :, None] * e[2][i][None, None, :]
    return dens


def _grid(case, gen):
    """opaque: the benchmark's scenes (amplitudes 5 to 20, clipped by the renderer); soft:
    a grid in the middle of training, opacities mostly below 1 and some values outside
    [0,1], as an unconstrained optimiser leaves them."""
    dims = (case["x"], case["y"], case["z"])
    pd = _pd(case)
    g = torch.empty(*dims, 4, device=DEV)
    g[..., :3] = torch.sigmoid(torch.randn(*dims, 3, generator=gen, device=DEV))
    if case.get("alpha", "soft") == "opaque":
        g[..., 3] = _blobs(dims, pd, 16 if max(dims) <= 300 else 64, gen, 5.0, 20.0)
    else:
        g[..., 3] = _blobs(dims, pd, 8, gen, 0.005, 0.06)
        wild = torch.rand(*dims, generator=gen, device=DEV) < 0.02
        g[wild] = torch.rand(int(wild.sum()), 4, generator=gen, device=DEV) * 2.0 - 0.5
    return g.to(DTYPES[case.get("dtype", "f32")])


def _cameras(count, rng):
    out = np.zeros((count, 4, 4), np.float32)
    for i in range(count):
        p = rng.standard_normal(3)
        p[2] = abs(p[2]) + 0.1
        p = 4.0 * p / np.linalg.norm(p)
        back = p / np.linalg.norm(p)
        x = np.cross([0.0, 0.0, 1.0] if abs(back[2]) < 0.999 else [0.0, 1.0, 0.0], back)
        x /= np.linalg.norm(x)
        y = np.cross(back, x)
        out[i, :3, 0], out[i, :3, 1], out[i, :3, 2], out[i, :3, 3] = x, y, back, p
        out[i, 3, 3] = 1.0
    return torch.from_numpy(out).to(DEV)


def _images(count, side, gen):
    """Smooth premultiplied pictures: colour noise over a soft disc, clear corners."""
    low = torch.rand(count, 4, 9, 9, generator=gen, device=DEV)
    img = torch.nn.functional.interpolate(low, size=(side, side), mode="bilinear", align_corners=True)
    a = torch.linspace(-1, 1, side, device=DEV)
    r = (a[:, None] ** 2 + a[None] ** 2).sqrt()
    alpha = (1.5 - 1.8 * r).clamp(0, 1)
    img = img.permute(0, 2, 3, 1).contiguous()
    img[..., 3] = alpha
    img[..., :3] *= alpha[..., None]
    return img.contiguous()


def _rays(count, cameras, gen, rng):
    """Rays of random pixels of several cameras, started at the near distance: (origins,
    directions, targets), camera after camera as a training batch has them."""
    T = _cameras(cameras, rng)
    own = (torch.arange(count, device=DEV) * cameras) // max(1, count)
    uv = torch.rand(count, 2, generator=gen, device=DEV) - 0.5
    C = T[own]
    d = FOV * uv[:, :1] * C[:, :3, 0] - FOV * uv[:, 1:] * C[:, :3, 1] - C[:, :3, 2]
    d = (d / d.norm(dim=1, keepdim=True)).contiguous()
    o = (C[:, :3, 3] + NEAR * d).contiguous()
    target = torch.rand(count, 4, generator=gen, device=DEV)
    target[:, :3] *= target[:, 3:]
    return o, d, target.contiguous()


def _generators(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 13)
    return gen, np.random.default_rng(int(seed) + 101)


def _scene_list(case):
    """(side, rays) of each scene of a batched case; the same for every seed."""
    rng = np.random.default_rng(case["scenes"] * 1000 + case["samples"])
    sides = [int(s) for s in case["sides"].split(",")]
    out = []
    for _ in range(case["scenes"]):
        n = int(round(math.exp(rng.uniform(math.log(case["min_rays"]), math.log(case["max_rays"])))))
        out.append((int(rng.choice(sides)), n))
    return out


def _batched_inputs(case, seed):
    gen, rng = _generators(case, seed)
    scs, o, d, t, own = [], [], [], [], []
    for i, (side, n) in enumerate(_scene_list(case)):
        pd = 3.0 / side
        dens = _blobs((side,) * 3, pd, 8, gen, 5.0, 20.0)
        sub = dens.flatten()[torch.randint(0, dens.numel(), (1 << 18,), generator=gen, device=DEV)]
        occ = dens > torch.quantile(sub, 0.95)   # 5 % of the cells
        cells = torch.cat([torch.rand(side, side, side, 3, generator=gen, device=DEV), dens[..., None]], -1)
        cells[~occ] = 0.0
        scs.append((cells.to(DTYPES[case["dtype"]]).contiguous(), occ, pd))
        oi, di, ti = _rays(n, 4, gen, rng)
        o.append(oi); d.append(di); t.append(ti)
        own.append(torch.full((n,), i, dtype=torch.int32, device=DEV))
    return scs, torch.cat(o), torch.cat(d), torch.cat(t), torch.cat(own)


def _moments(grid, gen):
    """Adam's moments and the |grad| sum of a run in progress."""
    m = 1e-6 * torch.randn(grid.shape, generator=gen, device=DEV)
    s = (2e-6 * (0.5 + torch.rand(grid.shape, generator=gen, device=DEV))) ** 2
    # cells that no ray has reached so far: the outer tenth of the box on each side
    seen = torch.ones(grid.shape[:3], dtype=torch.bool, device=DEV)
    for ax, n in enumerate(grid.shape[:3]):
        k = n // 10
        seen.narrow(ax, 0, k).zero_()
        seen.narrow(ax, n - k, k).zero_()
    m *= seen[..., None]
    s *= seen[..., None]
    return m, s, 100.0 * s.sqrt()


def prepare(case, seed):
    kind = case["kind"]
    gen, rng = _generators(case, seed)
    st = dict(case=case)
    if kind == "batched":
        scs, o, d, t, own = _batched_inputs(case, seed)
        scenes = [Scene(c, occ, pd, case["samples"], (FAR - NEAR) / case["samples"]) for c, occ, pd in scs]
        # the tile that the autotuner picks on such batches
        st["step"] = BatchedTrainStep(scenes, o.shape[0], mode=case["mode"], tiles=(1, 256, 1))
        st["rays"] = (o, d, t, own)
        return st
    grid = _grid(case, gen)
    pd = _pd(case)
    if kind == "clean":
        # stray cells: scattered opaque specks in an otherwise empty surround
        dims = grid.shape[:3]
        solid = _blobs(dims, pd, 4, gen, 0.5, 2.0, width=0.2)
        specks = torch.rand(dims, generator=gen, device=DEV)
        grid[..., 3] = torch.where(specks < 0.02, torch.rand(dims, generator=gen, device=DEV),
                                   torch.where(solid > 0.2, solid.clamp(max=1.0), torch.zeros_like(solid)))
        st["grid"] = grid
        return st
    if kind == "images":
        st.update(grid=grid, T=_cameras(case["cameras"], rng))
        return st
    delta = (FAR - NEAR) / case["samples"]
    st.update(delta=delta, pd=pd)
    if kind == "dropin":
        T = _cameras(case["cameras"], rng)
        st.update(grid=grid.requires_grad_(True), T=T, imgs=_images(case["cameras"], case["image"], gen),
                  coords=pg.generate_grid(case["x"], case["y"], case["z"], pd, device=DEV)[0],
                  delta=FAR / case["samples"], seed=int(seed))
        return st
    if kind == "step_cameras":
        st.update(T=_cameras(case["cameras"], rng), imgs=_images(case["cameras"], case["image"], gen),
                  ray_seed=1000 + int(seed))
        st["step"] = pg.FusedTrainStep(grid, pd, case["samples"], delta, mode=case["mode"], stratified=True,
                                       seed=STRAT_SEED, overlap_zero=case["zeroing"] == "marked",
                                       zeroing=case["zeroing"])
        return st
    st["o"], st["d"], st["target"] = _rays(case["rays"], min(100, case["rays"]), gen, rng)
    if kind == "render":
        st["grid"] = grid
    elif kind == "autograd":
        st["grid"] = grid.requires_grad_(True)
    elif kind == "step_rays":
        st["step"] = pg.FusedTrainStep(grid, pd, case["samples"], delta, mode=case["mode"], stratified=True,
                                       seed=STRAT_SEED, transmittance=case["transmittance"],
                                       overlap_zero=case["zeroing"] == "marked", zeroing=case["zeroing"])
    else:
        more = {}
        if kind == "growing":  # one receptive field of the schedule, held
            more = dict(progressive_growing=True, fields=[case["field"]], steps_per_field=1 << 30)
        tr = pg.Trainer(grid, pd, case["samples"], delta, ADAM["lr"], tv=case["tv"], beta=case["beta"],
                        mode=case["mode"], betas=ADAM["betas"], eps=ADAM["eps"], **more)
        for buf, val in zip((tr.opt.exp_avg, tr.opt.exp_avg_sq, tr.opt.abs_grad), _moments(grid, gen)):
            buf.copy_(val)   # as a resumed run loads them
        tr.opt.step_count = MOMENT_STEPS
        st["trainer"] = tr
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "render":
        with torch.no_grad():
            return pg.render_rays(st["grid"], st["o"], st["d"], st["delta"], case["samples"], st["pd"],
                                  mode=case["mode"],
                                  background=(1.0, 1.0, 1.0) if case["background"] else None)
    if kind == "autograd":
        g = st["grid"]
        g.grad = None
        px = pg.render_rays(g, st["o"], st["d"], st["delta"], case["samples"], st["pd"], mode=case["mode"],
                            background=(1.0, 1.0, 1.0) if case["background"] else None)
        torch.nn.functional.mse_loss(px, st["target"]).backward()
        return px, g.grad
    if kind == "step_rays":
        loss = st["step"].step_rays(st["o"], st["d"], st["target"])
        return loss, st["step"].grad
    if kind == "step_cameras":
        loss = st["step"].step_cameras(st["T"], st["imgs"], FOV, case["rays"], st["ray_seed"], near=NEAR)
        return loss, st["step"].grad
    if kind in ("trainer", "growing"):
        tr = st["trainer"]
        losses = tr.step_rays(st["o"], st["d"], st["target"])
        return losses, tr.grid, tr.opt.exp_avg, tr.opt.exp_avg_sq, tr.opt.abs_grad
    if kind == "batched":
        step = st["step"]
        step.set_rays(*st["rays"])
        loss = step.step()
        return loss, [sc.grad for sc in step.scenes]
    if kind == "dropin":
        g, T = st["grid"], st["T"]
        g.grad = None
        S, C, R = case["samples"], case["cameras"], case["per_camera"]
        torch.manual_seed(st["seed"])   # the pixels are drawn with torch.rand: the same ones in every pass
        samples, target, _, _ = pg.sample_camera_rays_batched(T, FOV, st["imgs"], R, S, st["delta"], False,
                                                              False, device=DEV)
        n = pg.normalize_samples_for_indecies(st["coords"], samples, st["pd"])
        if case["mode"] == "nearest":
            vals, mask = pg.get_nearest_voxels(n, g, clip=True)
        else:
            mask = pg.find_out_of_bound(n, g)
            corners = pg.get_grid_points_indices(n)
            pg.fix_out_of_bounds(corners.view(-1, 3), g)
            vals = pg.trilinear_interpolation(n, corners, g, clip=True)
        vals = vals * mask.unsqueeze(-1)
        px = pg.compute_alpha_weighted_pixels(vals.reshape(C, R, S, 4)).reshape(-1, 4)
        torch.nn.functional.mse_loss(px, target).backward()
        return px, g.grad
    if kind == "images":
        return render_camera_images(st["grid"], st["T"], case["image"], case["image"], FOV, NEAR,
                                    (FAR - NEAR) / case["samples"], case["samples"], _pd(case),
                                    mode=case["mode"])
    return pg.convolve_grid_to_remove_noise(st["grid"].clone(), kernel_size=case["kernel"],
                                            threshold=case["threshold"])


# ------------------------------------------------------------------------------- floors
def work(case):
    """Bytes and operations a pass cannot do without. A ray's samples are in bounds for
    about 0.7 of its length; trilinear samples read about four cells each that no other
    sample of the batch reads."""
    kind = case["kind"]
    if kind == "batched":
        b = f = 0.0
        cell = 8 if case["dtype"] == "bf16" else 16
        for side, n in _scene_list(case):
            occupied = 0.05 * side ** 3
            b += occupied * (cell + 16) + 60 * n
            f += 0.1 * n * case["samples"] * 250
        return dict(bytes=b, flops=f)
    G = case["x"] * case["y"] * case["z"]
    if kind == "clean":
        return dict(bytes=G * 48.0, flops=20.0 * G * 7)
    per, ops = (1, 40) if case["mode"] == "nearest" else (4, 180)
    cell = 8 if case.get("dtype") == "bf16" else 16
    if kind == "images":
        R = case["cameras"] * case["image"] ** 2
        return dict(bytes=min(G, 0.7 * R * case["samples"] * per) * cell + 16.0 * R,
                    flops=0.7 * R * case["samples"] * ops)
    R = case["cameras"] * case["per_camera"] if kind == "dropin" else case["rays"]
    N = 0.7 * R * case["samples"]
    touched = min(G, N * per)
    if kind == "render":
        return dict(bytes=touched * cell + 40.0 * R, flops=N * ops)
    flops = 2 * N * ops
    if kind in ("trainer", "growing"):
        # parameters, two moments and the |grad| sum read and written
        return dict(bytes=G * 128.0 + 56.0 * R, flops=flops + 40.0 * G)
    if kind in ("step_rays", "step_cameras") and case["zeroing"] == "marked":
        return dict(bytes=touched * (cell + 16) + 56.0 * R, flops=flops)
    return dict(bytes=touched * cell + G * 16.0 + 56.0 * R, flops=flops)


# ------------------------------------------------------------------------------- exact
# Sample positions are part of the interface: they are single-precision numbers, rounded
# after every operation, and they decide which cell a sample falls in. Below they are made
# that way; from the positions on, everything is in 64 bits.

def _mix(z):
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _stream(seed, a):
    with np.errstate(over="ignore"):
        return _mix(_mix(np.asarray([seed], np.uint64)) ^ a.astype(np.uint64))


def _unit(h, b):
    with np.errstate(over="ignore"):
        v = _mix(h ^ np.asarray(b, np.uint64)) >> np.uint64(40)
    return (v.astype(np.float64) * 2.0 ** -24).astype(np.float32)


def _jitter(rows, S):
    h = _stream(STRAT_SEED, rows)
    return torch.from_numpy(_unit(h[:, None], np.arange(S)[None])).to(DEV)


def _f32(v):
    return torch.tensor(v, dtype=torch.float32, device=DEV)


def _origin(shape, pd):
    return [float(np.float32(1 - math.ceil(s / 2)) * np.float32(pd)) for s in shape[:3]]


def _coords(o, d, S, delta, jitter, origin, pd):
    """[R,S,3] normalised positions in single precision, rounded operation by operation."""
    k = torch.arange(1, S + 1, device=DEV, dtype=torch.float32)[None].expand(o.shape[0], S)
    if jitter is not None:
        k = k - jitter
    t = _f32(delta) * k
    p = d[:, None, :] * t[..., None]
    p = o[:, None, :] + p
    return (p - _f32(origin)) / _f32(pd).expand_as(p)


def _camera_rays(T, uv):
    """Directions of the rays at uv [C,R,2] in single precision: the norm of a direction is
    accumulated with fused multiply-adds (formed here from 64-bit products)."""
    def plain(v):
        return ((v[..., 0] * v[..., 0] + v[..., 1] * v[..., 1]) + v[..., 2] * v[..., 2]).sqrt()
    x, y, z = T[:, :3, 0], T[:, :3, 1], -T[:, :3, 2]
    aspect = plain(x) / plain(y)
    one = torch.ones_like(aspect)
    u = _f32(FOV) * (uv[..., 0] - 0.5)
    v = -((_f32(FOV) * (one / aspect))[:, None] * (uv[..., 1] - 0.5))
    e = u[..., None] * x[:, None]
    e = e + v[..., None] * y[:, None]
    e = e + z[:, None]
    q = e.double()
    n = (q[..., 0] * q[..., 0]).float()
    n = (q[..., 1] * q[..., 1] + n.double()).float()
    n = (q[..., 2] * q[..., 2] + n.double()).float().sqrt()
    return e / n[..., None].expand_as(e)


def _corners(n, dims, mode):
    """[(cell index [..], weight [..])] of the samples at n, and their in-bounds mask."""
    X, Y, Z = dims
    size = torch.tensor(dims, device=DEV)
    if mode == "nearest":
        i = torch.round(n).long()
        inb = ((i >= 0) & (i < size)).all(-1)
        i = i % size
        return [((i[..., 0] * Y + i[..., 1]) * Z + i[..., 2], None)], inb
    inb = ((n >= 0) & (n < size)).all(-1)
    fl = torch.floor(n)
    f, c = fl.long() % size, torch.ceil(n).long() % size
    w = (n - torch.trunc(n)).double()
    out = []
    for corner in range(8):
        idx, wt = 0, 1.0
        for ax, (bit, s) in enumerate(((4, Y * Z), (2, Z), (1, 1))):
            low = bool(corner & bit)
            idx = idx + (f if low else c)[..., ax] * s
            wt = wt * ((1 - w[..., ax]) if low else w[..., ax])
        out.append((idx, wt))
    return out, inb


def _values(flat, n, dims, mode):
    corners, inb = _corners(n, dims, mode)
    v = 0.0
    for idx, wt in corners:
        c = flat[idx].double().clamp(0, 1)
        v = v + (c if wt is None else c * wt[..., None])
    return v * inb[..., None], corners, inb


def _scatter(grad, flat, corners, inb, dv, occ=None):
    dv = dv * inb[..., None]
    for idx, wt in corners:
        raw = flat[idx].double()
        g = torch.where((raw >= 0) & (raw <= 1), dv if wt is None else dv * wt[..., None], 0.0)
        if occ is not None:
            g = g * occ[idx][..., None]
        grad.index_add_(0, idx.reshape(-1), g.reshape(-1, 4))


def _composite(v):
    a = v[..., 3]
    T = torch.cumprod(torch.cat([torch.ones_like(a[:, :1]), 1 - a[:, :-1]], 1), 1)
    w = a * T
    return torch.cat([(v[..., :3] * w[..., None]).sum(1), w.sum(1, keepdim=True)], 1)


def _exact_pixels(flat, dims, coords_of, R, S, mode, background=None):
    out = torch.empty(R, 4, dtype=torch.float64, device=DEV)
    step = max(1, (1 << 20) // S)
    for lo in range(0, R, step):
        rows = torch.arange(lo, min(R, lo + step), device=DEV)
        v, _, _ = _values(flat, coords_of(rows), dims, mode)
        px = _composite(v)
        if background is not None:
            px = torch.cat([px[:, :3] + (1 - px[:, 3:]) * background, px[:, 3:]], 1)
        out[rows] = px
    return out


def _exact_step(flat, dims, coords_of, target, R, S, mode, background=None, beta=0.0, occ=None,
                grad=None, total=None):
    """(pixels, MSE, beta term, dense gradient [G,4]) of a training step in 64 bits."""
    if grad is None:
        grad = torch.zeros(flat.shape[0], 4, dtype=torch.float64, device=DEV)
    total = total or R
    px_out = torch.empty(R, 4, dtype=torch.float64, device=DEV)
    mse = torch.zeros((), dtype=torch.float64, device=DEV)
    bsum = torch.zeros((), dtype=torch.float64, device=DEV)
    step = max(1, (1 << 20) // S)
    for lo in range(0, R, step):
        rows = torch.arange(lo, min(R, lo + step), device=DEV)
        v, corners, inb = _values(flat, coords_of(rows), dims, mode)
        v = v.requires_grad_(True)
        px = _composite(v)
        if background is not None:
            px = torch.cat([px[:, :3] + (1 - px[:, 3:]) * background, px[:, 3:]], 1)
        part = ((px - target[rows].double()) ** 2).sum() / (4.0 * total)
        loss = part
        if beta:
            a = v[..., 3]
            b = beta * (torch.log(a + BETA_EPS) - torch.log(1 - a + BETA_EPS)).sum() / (float(R) * S)
            bsum += b.detach()
            loss = loss + b
        (dv,) = torch.autograd.grad(loss, v)
        mse += part.detach()
        px_out[rows] = px.detach()
        _scatter(grad, flat, corners, inb, dv, occ)
    return px_out, mse, bsum, grad


def _tv(grid):
    """(sum of squared neighbour differences, its gradient over 2) in 64 bits."""
    q, g = 0.0, torch.zeros(grid.shape, dtype=torch.float64, device=DEV)
    for ax in range(3):
        n = grid.shape[ax] - 1
        diff = grid.narrow(ax, 0, n).double() - grid.narrow(ax, 1, n).double()
        q = q + (diff ** 2).sum()
        g.narrow(ax, 0, n).add_(diff)
        g.narrow(ax, 1, n).sub_(diff)
    return q, g


def _adam(p, g, m, s):
    b1, b2 = ADAM["betas"]
    t = MOMENT_STEPS + 1
    m = b1 * m.double() + (1 - b1) * g
    s = b2 * s.double() + (1 - b2) * g * g
    p = p.double() - ADAM["lr"] / (1 - b1 ** t) * m / (s.sqrt() / math.sqrt(1 - b2 ** t) + ADAM["eps"])
    return p, m, s


def exact(case, seed):
    kind = case["kind"]
    gen, rng = _generators(case, seed)
    if kind == "batched":
        scs, o, d, t, own = _batched_inputs(case, seed)
        S, R = case["samples"], o.shape[0]
        mse, grads = 0.0, []
        for i, (cells, occ, pd) in enumerate(scs):
            rows = (own == i).nonzero().reshape(-1)
            oi, di, ti = o[rows], d[rows], t[rows]
            org = _origin(cells.shape, pd)
            _, part, _, g = _exact_step(
                cells.reshape(-1, 4), tuple(cells.shape[:3]),
                lambda r: _coords(oi[r], di[r], S, (FAR - NEAR) / S, None, org, pd),
                ti, rows.numel(), S, case["mode"], occ=occ.reshape(-1).double(), total=R)
            mse = mse + part
            grads.append(g.reshape(cells.shape))
        return mse, grads
    grid = _grid(case, gen)
    pd, dims = _pd(case), (case["x"], case["y"], case["z"])
    org = _origin(dims, pd)
    if kind == "clean":
        return None   # cells are kept or cleared: nothing is rounded into them
    S = case["samples"]
    delta = (FAR - NEAR) / S
    flat = grid.reshape(-1, 4)
    if kind == "images":
        T, H = _cameras(case["cameras"], rng), case["image"]
        at = torch.arange(H, device=DEV, dtype=torch.float32) / H
        uv = torch.stack([at.expand(H, H), at[:, None].expand(H, H)], -1).reshape(1, H * H, 2)
        out = []
        for c in range(case["cameras"]):
            dirs = _camera_rays(T[c:c + 1], uv)[0]
            o = T[c, :3, 3] + NEAR * dirs
            px = _exact_pixels(flat, dims, lambda r: _coords(o[r], dirs[r], S, delta, None, org, pd),
                               H * H, S, case["mode"])
            out.append(px.reshape(H, H, 4))
        return torch.stack(out)
    if kind == "dropin":
        T, imgs = _cameras(case["cameras"], rng), _images(case["cameras"], case["image"], gen)
        C, Rc, H = case["cameras"], case["per_camera"], case["image"]
        torch.manual_seed(int(seed))
        uv = torch.rand(C, Rc, 2, device=DEV)
        dirs = _camera_rays(T, uv).reshape(-1, 3)
        o = T[:, None, :3, 3].expand(C, Rc, 3).reshape(-1, 3)
        pix = (_f32(H) * uv).round().clamp(max=H - 1).long()
        cam = torch.arange(C, device=DEV)[:, None].expand(C, Rc)
        target = imgs[cam, pix[..., 1], pix[..., 0]].reshape(-1, 4)
        px, _, _, g = _exact_step(flat, dims, lambda r: _coords(o[r], dirs[r], S, FAR / S, None, org, pd),
                                  target, C * Rc, S, case["mode"])
        return px, g.reshape(grid.shape)
    if kind == "step_cameras":
        T, imgs = _cameras(case["cameras"], rng), _images(case["cameras"], case["image"], gen)
        R, C, H = case["rays"], case["cameras"], case["image"]
        h = _stream(1000 + int(seed), np.arange(R))
        uv = torch.from_numpy(np.stack([_unit(h, 0), _unit(h, 1)], -1)).to(DEV)
        cam = (torch.arange(R, device=DEV) * C) // R
        dirs = _camera_rays(T[cam], uv[:, None])[:, 0]
        o = T[cam][:, :3, 3] + NEAR * dirs
        pix = (_f32(H) * uv).round().clamp(max=H - 1).long()
        target = imgs[cam, pix[:, 1], pix[:, 0]]
        jit = _jitter(np.arange(R), S)
        _, mse, _, g = _exact_step(flat, dims, lambda r: _coords(o[r], dirs[r], S, delta, jit[r], org, pd),
                                   target, R, S, case["mode"])
        return mse, g.reshape(grid.shape)
    o, d, target = _rays(case["rays"], min(100, case["rays"]), gen, rng)
    R = case["rays"]
    white = 1.0 if case.get("background") else None
    if kind == "render":
        return _exact_pixels(flat, dims, lambda r: _coords(o[r], d[r], S, delta, None, org, pd), R, S,
                             case["mode"], white)
    if kind == "autograd":
        px, _, _, g = _exact_step(flat, dims, lambda r: _coords(o[r], d[r], S, delta, None, org, pd), target,
                                  R, S, case["mode"], white)
        return px, g.reshape(grid.shape)
    if kind == "step_rays":
        _, mse, _, g = _exact_step(
            flat, dims, lambda r: _coords(o[r], d[r], S, delta, _jitter(r.cpu().numpy(), S), org, pd),
            target, R, S, case["mode"])
        return mse, g.reshape(grid.shape)
    # trainer, growing
    m, s, acc = _moments(grid, gen)
    if kind == "trainer":
        _, mse, beta, g = _exact_step(flat, dims, lambda r: _coords(o[r], d[r], S, delta, None, org, pd),
                                      target, R, S, case["mode"], beta=case["beta"])
        g = g.reshape(grid.shape)
        shown = grid
    else:
        w = case["field"]
        stride, start = max(1, w // 4), w // 2
        x = grid.double().permute(3, 0, 1, 2)[None]
        small64 = torch.nn.functional.avg_pool3d(x, (w,) * 3, stride=stride)[0].permute(1, 2, 3, 0).contiguous()
        sdims = tuple(small64.shape[:3])
        # coordinate of the pooled grid's first cell, in single precision
        sorg = [float(np.float32(start - math.ceil(n / 2) + 1) * np.float32(pd)) for n in dims]
        _, mse, beta, g = _exact_step(small64.reshape(-1, 4), sdims,
                                      lambda r: _coords(o[r], d[r], S, delta, None, sorg, pd * stride),
                                      target, R, S, case["mode"], beta=case["beta"])
        g = g.reshape(small64.shape)
        shown = small64
    tv = torch.zeros((), dtype=torch.float64, device=DEV)
    if case["tv"] > 0 and (kind == "trainer" or case["field"] < 19):
        q, tg = _tv(shown)
        tv = case["tv"] * q.sqrt()
        g = g + case["tv"] / q.sqrt() * tg
    if kind == "growing":
        g = _unpool(g, dims, case["field"])
    p, m, s = _adam(grid, g, m, s)
    return torch.stack([mse, tv, beta]), p, m, s, acc.double() + g.abs()


def _unpool(g, dims, w):
    """The adjoint of the average pooling, one axis after the other."""
    stride = max(1, w // 4)
    for ax in range(3):
        shape = list(g.shape)
        shape[ax] = dims[ax]
        out = torch.zeros(shape, dtype=torch.float64, device=DEV)
        for k in range(w):
            at = torch.arange(g.shape[ax], device=DEV) * stride + k
            out.index_add_(ax, at, g)
        g = out
    return g / float(w) ** 3
