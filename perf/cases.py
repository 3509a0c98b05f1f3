"""What a user of this library has it do, as measurable cases through its public entry points.

A case is a dict of plain values; `prepare` makes what the user's program holds before the call
(inputs on the GPU, contexts, buffers, a trainer), `run` is one pass, `work` the bytes and
operations the pass cannot do without, `exact` the outputs in 64-bit arithmetic where they are
computed numbers. Sizes follow the library's workloads: 5 cascades of 128^3 with 2^14 rays and
2^18 samples a step, compositor batches of up to 2^22 samples, a 16 x 2^19 x 2 hash grid, sixteen
scenes of 2^10 to 2^16 rays, 800 x 800 frames.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from turbonerf_b200 import autograd, hotpath as hp, scenes
from turbonerf_b200.renderer import Camera, CUDARenderBuffer, Renderer, RenderRequest
from turbonerf_b200.trainer import BoundingBox, Dataset, SyntheticNeRF, Trainer

DEV = "cuda"
DT_MIN = float(scenes.MIN_STEP_SIZE)
NO_CUT = 0xFFFFFFFF
THRESHOLD = 0.01   # density above which a cell is occupied
LAMBDA = 1e-3      # distortion loss weight
N_MLP = 7168
# samples a ray of the marched scenes finds, by cascade count: the mean and a safe capacity
MEAN_SAMPLES = {1: 1020, 2: 640, 3: 420, 4: 228, 5: 195}
CAP_SAMPLES = {1: 1024, 2: 800, 3: 560, 4: 320, 5: 280}
MULTI_MEAN, MULTI_CAP = 100, 200


# ---- the cases ---------------------------------------------------------------------------
def listed():
    return [
        # a handful of rays through one cascade at a fixed step: an interactive probe or a preview
        # patch, where launches and latency are everything
        dict(name="march_small", kind="march", rays=256, cascades=1, batch=0),
        # the march of every training step: clip, count, batch cut, emit
        dict(name="march_train", kind="march", rays=1 << 14, cascades=5, batch=1 << 18),
        # many scenes trained or evaluated together, each with its own grid, uneven ray counts
        dict(name="march_multi_scene", kind="multi", scenes=16, ray_lo=1 << 10, ray_hi=1 << 16),
        # differentiable volume rendering inside a torch program: a small patch of rays
        dict(name="volume_render_small", kind="volume", samples=5000, mean=48, activation=0),
        # the same on a full-image batch, forward and backward, compositor and distortion loss
        dict(name="volume_render_large", kind="volume", samples=1 << 22, mean=64, activation=0),
        # everything between the network's forward and backward in one training step
        dict(name="train_losses", kind="losses", samples=1 << 18, mean=48, activation=1),
        # the occupancy grid's update after a step: query points, decay, max-update, bitfield
        dict(name="occupancy_update", kind="occupancy", cascades=5, resolution=128, updates=1 << 16, all=False),
        # the optimizer step over a hash grid of which a batch touched half the entries
        dict(name="adam_step", kind="adam", grid=16 << 20, mlp=N_MLP, touched=0.5),
        # the hash-grid encoding of one step's samples, forward and backward
        dict(name="hashgrid", kind="hashgrid", samples=1 << 18, levels=16, log2_table=19),
        # a whole training step of the built-in scene, enqueued as a training loop does
        dict(name="train_step", kind="trainer", rays=1 << 14, batch=1 << 18, updates=1 << 16),
        # a whole training step on posed images with the hash-grid network, metrics read each step
        dict(name="train_step_images", kind="image_trainer", rays=1 << 14, batch=1 << 18, updates=1 << 16,
             images=24, size=400),
        # a frame of the trained scene
        dict(name="render_frame", kind="render", width=800, height=800, budget=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["march", "march", "multi", "volume", "volume", "losses", "occupancy", "adam", "hashgrid",
                       "hashgrid", "trainer", "image_trainer", "render"])
    if kind == "march":
        cascades = rng.randint(1, 5)
        rays = _log_int(rng, 64, 1 << (11 + cascades))
        batch = rng.choice([0, _log_int(rng, max(4096, 4 * rays), 1 << 19)])
        return dict(kind=kind, rays=rays, cascades=cascades, batch=batch)
    if kind == "multi":
        lo = _log_int(rng, 64, 1 << 10)
        return dict(kind=kind, scenes=rng.randint(2, 16), ray_lo=lo, ray_hi=_log_int(rng, 4 * lo, 1 << 15))
    if kind == "volume":
        return dict(kind=kind, samples=_log_int(rng, 1 << 10, 1 << 22), mean=_log_int(rng, 4, 128),
                    activation=rng.randint(0, 1))
    if kind == "losses":
        return dict(kind=kind, samples=_log_int(rng, 1 << 12, 1 << 21), mean=_log_int(rng, 8, 128),
                    activation=rng.randint(0, 1))
    if kind == "occupancy":
        return dict(kind=kind, cascades=rng.randint(1, 5), resolution=rng.choice([64, 128, 128]),
                    updates=_log_int(rng, 1 << 10, 1 << 20), all=rng.choice([False, True]))
    if kind == "adam":
        return dict(kind=kind, grid=_log_int(rng, 1 << 14, 16 << 20), mlp=_log_int(rng, 64, 1 << 14),
                    touched=round(rng.uniform(0.02, 1.0), 3))
    if kind == "hashgrid":
        return dict(kind=kind, samples=_log_int(rng, 1 << 10, 1 << 18), levels=rng.randint(4, 16),
                    log2_table=rng.randint(14, 19))
    if kind == "render":
        return dict(kind=kind, width=_log_int(rng, 48, 800), height=_log_int(rng, 48, 800),
                    budget=rng.choice([0, 1 << 20]))
    rays = _log_int(rng, 1 << 11, 1 << 14)
    c = dict(kind=kind, rays=rays, batch=_log_int(rng, 1 << 15, 1 << 18), updates=_log_int(rng, 1 << 12, 1 << 16))
    if kind == "image_trainer":
        c.update(images=rng.randint(4, 32), size=_log_int(rng, 64, 400))
    return c


# ---- inputs ------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _field(seed, n_blobs=8):
    return scenes.make_blob_field(np.random.default_rng(seed), n_blobs)


def _grid(fld, n_levels, base, resolution=128):
    """Densities [levels][R^3] of the blob field at the cell centres (Morton order) and the
    bitfield of those above the threshold."""
    V = resolution ** 3
    m = torch.arange(V, device=DEV, dtype=torch.int64)

    def compact(v):
        v = v & 0x09249249
        v = (v | (v >> 2)) & 0x030C30C3
        v = (v | (v >> 4)) & 0x0300F00F
        v = (v | (v >> 8)) & 0x030000FF
        return (v | (v >> 16)) & 0x000003FF

    unit = [(compact(m >> c).float() - resolution / 2 + 0.5) / resolution for c in range(3)]
    density = torch.zeros((n_levels, V), device=DEV)
    bits = torch.zeros(V, dtype=torch.uint8, device=DEV)
    for k in range(n_levels):
        ls = base * (1 << k)
        for cx, cy, cz, sd, pk in fld.blobs.astype(np.float64).tolist():
            d2 = (unit[0] * ls - cx) ** 2 + (unit[1] * ls - cy) ** 2 + (unit[2] * ls - cz) ** 2
            density[k] += pk * torch.exp(d2 * (-0.5 / (sd * sd)))
        bits |= (density[k] > THRESHOLD).to(torch.uint8) << k
    return density, bits


def _sphere_rays(g, n, radius, jitter=0.05):
    """Origins on a sphere, directions toward the centre with a little noise: [3 n] each."""
    o = torch.nn.functional.normalize(torch.randn((n, 3), device=DEV, generator=g), dim=1)
    d = torch.nn.functional.normalize(-o + jitter * torch.randn((n, 3), device=DEV, generator=g), dim=1)
    return (radius * o).t().contiguous().view(-1), d.t().contiguous().view(-1)


def _counts(g, total, mean):
    """Sample counts of round(total / mean) rays that add up to `total` (a random composition:
    geometric around the mean), with a tenth as many rays that met nothing in between, and the
    counts' exclusive scan."""
    live = max(1, min(total, round(total / mean)))
    cuts = torch.randperm(total - 1, device=DEV, generator=g)[:live - 1].sort()[0] + 1
    end = torch.tensor([total], device=DEV)
    c = torch.diff(torch.cat([end * 0, cuts, end]))
    R = live + live // 10
    at = torch.randperm(R, device=DEV, generator=g)[:live].sort()[0]
    counts = torch.zeros(R, dtype=torch.int64, device=DEV)
    counts[at] = c
    return counts, torch.cumsum(counts, 0) - counts


def _batch(seed, total, mean, activation):
    """A packed sample batch as a march and a network leave it."""
    g = _gen(seed)
    c, off = _counts(g, total, mean)
    R = c.numel()
    ray = torch.repeat_interleave(torch.arange(R, device=DEV), c)
    sigma = torch.randn(total, device=DEV, generator=g) * 2.0
    density = torch.exp(sigma).clamp(max=1e4) if activation == 0 else sigma + 1.0
    rgb = torch.sigmoid(torch.randn((3, total), device=DEV, generator=g))
    dt = (0.5 + 1.5 * torch.rand(total, device=DEV, generator=g)) * DT_MIN
    t0 = torch.rand(R, device=DEV, generator=g)
    end = torch.cumsum(dt.double(), 0)
    start = end - dt.double()
    excl = start - start[off.clamp_max(total - 1)][ray]
    t = (t0.double()[ray] + excl).float()
    m = t + 0.5 * dt
    last, first = (off + c - 1).clamp_min(0), off.clamp_max(total - 1)  # of rays with samples
    span = (t[last] + dt[last] - t[first]).clamp_min(1e-6)
    m_norm = ((m - t[first][ray]) / span[ray]).clamp(0.0, 1.0)
    dt_norm = dt / span[ray]
    target = torch.rand((4, R), device=DEV, generator=g)
    target[3] = 1.0
    bg = torch.rand((3, R), device=DEV, generator=g)
    return dict(counts=c.to(torch.int32), offsets=off.to(torch.int32), ray=ray, density=density.contiguous(), rgb=rgb,
                dt=dt, t=t, m_norm=m_norm, dt_norm=dt_norm, target=target, bg=bg,
                grad_rgba=torch.randn((4, R), device=DEV, generator=g),
                grad_dist=torch.rand(R, device=DEV, generator=g))


def _look_at(eye):
    eye = np.asarray(eye, np.float64)
    f = -eye / np.linalg.norm(eye)
    r = np.cross(f, [0.0, 1.0, 0.0])
    r /= np.linalg.norm(r)
    return np.stack([r, np.cross(f, r), f, eye], axis=1)


def _march_state(case, seed):
    n, levels = case["rays"], case["cascades"]
    single = levels == 1
    base = 3.0 if single else 1.0
    aabb = 3.0 if single else float(1 << (levels - 1))
    _, bits = _grid(_field(seed), levels, base)
    ori, dr = _sphere_rays(_gen(seed), n, 4.0)
    h = aabb / 2
    s = dict(n=n, bits=bits, ori=ori, dir=dr, bbox=(-h, -h, -h, h, h, h), inv=1.0 / aabb,
             grid=hp.GridSpec(levels, 128, base), batch=case["batch"] or NO_CUT, ctx=hp.Context(),
             march=hp.MarchSpec(0.0, DT_MIN, DT_MIN, 1024) if single else
             hp.MarchSpec(1.0 / 256.0, DT_MIN, float(np.float32(aabb) * np.float32(DT_MIN)), 0))
    s["n_steps"] = torch.zeros(n, dtype=torch.int32, device=DEV)
    s["info"] = torch.zeros(4, dtype=torch.int32, device=DEV)
    s["offsets"] = torch.zeros(n, dtype=torch.int32, device=DEV)
    s["stride"] = case["batch"] or n * CAP_SAMPLES[levels]
    s["samples"] = hp.alloc_samples(s["stride"], DEV)
    return s


def _march_count(s):
    t, t_max, alive = hp.rays_init_bbox(s["ori"], s["dir"], s["n"], s["n"], s["bbox"])
    hp.march_count(s["ctx"], s["grid"], s["bits"], s["bbox"], s["march"], s["n"], s["n"], s["ori"], s["dir"], t, t_max,
                   alive, s["batch"], n_steps=s["n_steps"], batch_info=s["info"])
    return t, alive


def _multi_rays(case):
    k, lo, hi = case["scenes"], case["ray_lo"], case["ray_hi"]
    return [int(lo * (hi / lo) ** ((i + 0.5) / k)) for i in range(k)]


def _multi_state(case, seed):
    rng = np.random.default_rng(seed)
    counts = _multi_rays(case)
    rng.shuffle(counts)
    levels = [1 + i % 5 for i in range(len(counts))]
    rng.shuffle(levels)
    R = sum(counts)
    g = _gen(seed)
    ori, dr = torch.empty((3, R), device=DEV), torch.empty((3, R), device=DEV)
    table, begin = [], 0
    for n, lv in zip(counts, levels):
        aabb = float(np.float32(math.exp(rng.uniform(math.log(0.5), math.log(16.0)))))
        fld = scenes.make_blob_field(rng, int(rng.integers(8, 33)))
        fld.blobs[:, :4] *= np.float32(aabb / 3.0)
        fld.blobs[:, 3] *= np.float32(0.3)  # a trained scene: surfaces fill a small part of the box
        base = float(np.float32(aabb) / np.float32(1 << (lv - 1)))
        _, bits = _grid(fld, lv, base)
        o, d = _sphere_rays(g, n, 4.0 * aabb / 3.0)
        ori[:, begin:begin + n] = o.view(3, n)
        dr[:, begin:begin + n] = d.view(3, n)
        h = aabb / 2
        table.append(dict(grid=hp.GridSpec(lv, 128, base), bitfield=bits, bbox=(-h, -h, -h, h, h, h),
                          march=hp.MarchSpec(1.0 / 256.0, DT_MIN, float(np.float32(max(aabb, 1.0)) *
                                                                        np.float32(DT_MIN)), 1024),
                          inv_aabb=1.0 / aabb, ray_begin=begin, n_rays=n))
        begin += n
    # the box clip of every scene's rays, as the march's inputs; alive flags are copied back each pass
    t, t_max = torch.zeros(R, device=DEV), torch.zeros(R, device=DEV)
    alive = torch.zeros(R, dtype=torch.uint8, device=DEV)
    for sc in table:
        b, n = sc["ray_begin"], sc["n_rays"]
        o, d = ori[:, b:b + n].contiguous().view(-1), dr[:, b:b + n].contiguous().view(-1)
        t[b:b + n], t_max[b:b + n], alive[b:b + n] = hp.rays_init_bbox(o, d, n, n, sc["bbox"])
    s = dict(R=R, ctx=hp.Context(), table=hp.scene_table(table), ori=ori.view(-1), dir=dr.view(-1), t=t, t_max=t_max,
             alive0=alive, alive=alive.clone(), n_steps=torch.zeros(R, dtype=torch.int32, device=DEV),
             offsets=torch.zeros(R, dtype=torch.int32, device=DEV),
             scene_samples=torch.zeros(len(table), dtype=torch.int32, device=DEV),
             info=torch.zeros(4, dtype=torch.int32, device=DEV))
    s["stride"] = R * MULTI_CAP
    s["samples"] = hp.alloc_samples(s["stride"], DEV)
    return s


def _multi_count(s):
    s["alive"].copy_(s["alive0"])
    hp.multi_march_count(s["ctx"], s["table"], s["R"], s["ori"], s["dir"], s["t"], s["t_max"], s["alive"],
                         n_steps=s["n_steps"], scene_samples=s["scene_samples"], info=s["info"])


def _adam_state(case, seed):
    g = _gen(seed)
    ng, nm = case["grid"], case["mlp"]
    n = ng + nm
    grad = torch.randn(n, device=DEV, generator=g) * 1e-3
    entry = torch.rand((ng + 1) // 2, device=DEV, generator=g) < case["touched"]  # both features of an entry
    grad[:ng] *= entry.repeat_interleave(2)[:ng]
    return dict(w=torch.rand(n, device=DEV, generator=g) * 2e-4 - 1e-4, g=grad, m=torch.zeros(n, device=DEV),
                v=torch.zeros(n, device=DEV), steps=torch.zeros(n, dtype=torch.int32, device=DEV), ng=ng, nm=nm)


def _occupancy_state(case, seed):
    g = _gen(seed)
    R, L, n = case["resolution"], case["cascades"], case["updates"]
    density, bits = _grid(_field(seed), L, 1.0, R)
    ri = lambda hi: torch.randint(0, hi, (n,), device=DEV, generator=g, dtype=torch.int32)  # noqa: E731
    return dict(grid=hp.GridSpec(L, R, 1.0), density=density.view(-1), bits=bits, levels=ri(L), cells=ri(R ** 3),
                rand3=torch.rand(3 * n, device=DEV, generator=g), n=n, inv=1.0 / (1 << (L - 1)),
                values=torch.randn(n, device=DEV, generator=g) * 3.0, select=torch.rand(n, device=DEV, generator=g),
                all=case["all"], ctx=hp.Context(), count=torch.zeros(1, dtype=torch.int32, device=DEV))


def _hashgrid_state(case, seed):
    """Positions along rays through the unit cube, as a march emits them."""
    g = _gen(seed)
    n = case["samples"]
    spec = hp.HashgridSpec(case["levels"], case["log2_table"], 16.0, math.exp(math.log(2048.0) / 15.0))
    n_rays = (n + 47) // 48
    o = torch.rand((n_rays, 3), device=DEV, generator=g)
    d = torch.nn.functional.normalize(torch.randn((n_rays, 3), device=DEV, generator=g), dim=1)
    k = torch.arange(48, device=DEV) * (DT_MIN / 2)
    pos = (o[:, None] + d[:, None] * k[None, :, None]).clamp(0.0, 1.0).view(-1, 3)[:n].t().contiguous()
    nh, _ = spec.n_params()
    return dict(spec=spec, n=n, pos=pos.view(-1), params=torch.rand(nh, device=DEV, generator=g) * 2e-4 - 1e-4,
                dfeat=torch.randn(spec.n_features * n, device=DEV, generator=g),
                feat=torch.zeros(spec.n_features * n, device=DEV), grads=torch.zeros(nh, device=DEV))


def _nerf(seed, levels=5, dataset=None):
    fld = _field(seed)
    density, bits = _grid(fld, levels, 1.0)
    return SyntheticNeRF(BoundingBox(float(1 << (levels - 1))), levels, fld.blobs, fld.waves, density.cpu().numpy(),
                         bits.cpu().numpy(), dataset=dataset)


def _trainer(case, seed, nerf, n_mlp=N_MLP, n_grid=16 << 20):
    tr = Trainer(nerf, n_rays_per_step=case["rays"], occupancy_cells_per_step=case["updates"],
                 distortion_lambda=LAMBDA, occupancy_threshold=THRESHOLD, n_grid_params=n_grid, n_mlp_params=n_mlp,
                 beta2=0.99, seed=seed & 0x7FFFFFFF)
    tr.use_distortion_loss = True
    tr.setup_data(batch_size=case["batch"])
    return tr


def _view(tr, which):
    """A view of one of the trainer's device buffers. It holds the trainer, which owns the memory:
    a view that outlives the other references must not outlive the buffer."""
    v = tr.buffer(which)
    v.owner = tr
    return v


def _dataset(case, seed):
    rng = np.random.default_rng(seed)
    n, px = case["images"], case["size"]
    cams = []
    for _ in range(n):
        e = rng.normal(size=3)
        cams.append(Camera((px, px), 0.1, 100.0, (1.4 * px, 1.4 * px), (px / 2, px / 2), (0.0, 0.0),
                           _look_at(4.0 * e / np.linalg.norm(e))))
    imgs = rng.integers(0, 256, (n, px, px, 4), dtype=np.uint8)
    imgs[..., 3] = np.where(rng.random((n, px, px)) < 0.4, 0, 255)
    return Dataset(cams, imgs)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind)
    if kind == "march":
        s.update(_march_state(case, seed))
    elif kind == "multi":
        s.update(_multi_state(case, seed))
    elif kind == "volume":
        b = _batch(seed, case["samples"], case["mean"], case["activation"])
        s.update(b, sigma=b["density"].requires_grad_(True), activation=case["activation"])
        s["rgb"].requires_grad_(True)
    elif kind == "losses":
        b = _batch(seed, case["samples"], case["mean"], case["activation"])
        R, S = b["counts"].numel(), case["samples"]
        s.update(b, R=R, S=S, ctx=hp.Context(), rb=hp.ray_batch(b["counts"], b["offsets"], R, R, S),
                 activation=case["activation"], grad=torch.zeros(S, device=DEV), drgb=torch.zeros(3 * S, device=DEV),
                 rgba=torch.zeros(4 * R, device=DEV), sums=torch.zeros(2, device=DEV))
    elif kind == "occupancy":
        s.update(_occupancy_state(case, seed))
    elif kind == "adam":
        s.update(_adam_state(case, seed))
    elif kind == "hashgrid":
        s.update(_hashgrid_state(case, seed))
    elif kind in ("trainer", "image_trainer"):
        if kind == "trainer":
            tr = _trainer(case, seed, _nerf(seed))
        else:
            spec = hp.HashgridSpec.reference(16.0)
            n_hash, n_head = spec.n_params()
            tr = _trainer(case, seed, _nerf(seed, dataset=_dataset(case, seed)), n_mlp=n_head, n_grid=n_hash)
            tr.use_hashgrid(spec)
        s.update(trainer=tr, weights=_view(tr, 0), grads=_view(tr, 1), m=_view(tr, 2), v=_view(tr, 3),
                 density=_view(tr, 5))
    elif kind == "render":
        w, h = case["width"], case["height"]
        tr = _trainer(dict(rays=4096, batch=1 << 16, updates=0), seed, _nerf(seed), n_grid=1 << 16)
        cam = Camera((w, h), 0.1, 100.0, (0.7 * w, 0.7 * w), (w / 2, h / 2), (0.0, 0.0), _look_at((0.3, 0.8, 4.0)))
        s.update(trainer=tr, renderer=Renderer(batch_size=case["budget"]),
                 request=RenderRequest(cam, [tr], CUDARenderBuffer()))
    else:
        raise ValueError(kind)
    return s


# ---- one pass ----------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "march":
        t, alive = _march_count(s)
        hp.march_emit(s["ctx"], s["grid"], s["bits"], s["bbox"], s["march"], s["inv"], s["n"], s["n"], s["stride"],
                      s["info"], s["ori"], s["dir"], t, alive, s["n_steps"], offsets=s["offsets"],
                      samples=s["samples"])
        return dict(s["samples"], ray_t=t, alive=alive, n_steps=s["n_steps"], offsets=s["offsets"], info=s["info"])
    if kind == "multi":
        _multi_count(s)
        hp.multi_march_emit(s["ctx"], s["table"], s["R"], s["stride"], s["ori"], s["dir"], s["t"], s["alive"],
                            s["n_steps"], samples=s["samples"], offsets=s["offsets"])
        return dict(s["samples"], alive=s["alive"], n_steps=s["n_steps"], offsets=s["offsets"],
                    scene_samples=s["scene_samples"], info=s["info"])
    if kind == "volume":
        rgba = autograd.composite(s["sigma"], s["rgb"], s["dt"], s["counts"], s["offsets"], activation=s["activation"])
        dist = autograd.distortion_loss(s["sigma"], s["m_norm"], s["dt_norm"], s["counts"], s["offsets"], LAMBDA,
                                        s["activation"])
        d_sigma, d_rgb = torch.autograd.grad([rgba, dist], [s["sigma"], s["rgb"]], [s["grad_rgba"], s["grad_dist"]])
        return dict(rgba=rgba, dist=dist, d_sigma=d_sigma, d_rgb=d_rgb)
    if kind == "losses":
        s["grad"].zero_()
        hp.train_losses(s["ctx"], s["rb"], s["density"], s["rgb"], s["dt"], s["m_norm"], s["dt_norm"], s["t"],
                        s["target"], s["bg"], s["grad"], inv_nrays=1.0 / s["R"], lam=LAMBDA,
                        activation=s["activation"], ray_rgba=s["rgba"], dL_drgb=s["drgb"], loss_sums=s["sums"])
        return dict(rgba=s["rgba"], grad=s["grad"], d_rgb=s["drgb"], sums=s["sums"])
    if kind == "occupancy":
        pos = hp.occupancy_sample_points(s["grid"], s["levels"], s["cells"], s["rand3"], s["n"], s["inv"])
        hp.occupancy_update(s["ctx"], s["grid"], s["density"], s["bits"], s["levels"], s["cells"], s["values"],
                            s["select"], activation=1, sample_all=s["all"], threshold=THRESHOLD,
                            n_occupied=s["count"])
        return dict(pos=pos, density=s["density"], bits=s["bits"], count=s["count"])
    if kind == "adam":
        hp.adam_step(s["w"], s["g"], s["m"], s["v"], s["steps"], s["ng"], s["nm"], 1e-2)
        return dict(w=s["w"], m=s["m"], v=s["v"], steps=s["steps"])
    if kind == "hashgrid":
        hp.hashgrid_encode(s["spec"], s["pos"], s["params"], s["n"], s["n"], out=s["feat"])
        s["grads"].zero_()
        hp.hashgrid_backward(s["spec"], s["pos"], s["dfeat"], s["grads"], s["n"], s["n"], touched=False)
        return dict(feat=s["feat"], grads=s["grads"])
    if kind == "trainer":
        s["trainer"].train_step_async()
        return dict(w=s["weights"], m=s["m"], v=s["v"], density=s["density"])
    if kind == "image_trainer":
        m = s["trainer"].train_step()
        return dict(loss=m.loss, n_rays=m.n_rays, n_samples=m.n_samples, grads=s["grads"], w=s["weights"],
                    density=s["density"])
    if kind == "render":
        stats = s["renderer"].submit(s["request"])
        return dict(rgba=s["request"].output.rgba, rays_hit=stats["rays_hit"], samples=stats["samples"])
    raise ValueError(kind)


# ---- what a pass cannot do without -----------------------------------------------------------
def work(case):
    """Bytes: every input read once, every output written once. Sample counts that only a march
    finds are estimated from the scenes' geometry."""
    kind = case["kind"]
    if kind == "march":
        n = case["rays"]
        smp = n * MEAN_SAMPLES[case["cascades"]]
        smp = min(smp, case["batch"]) if case["batch"] else smp
        return dict(bytes=n * (24 + 9 + 8) + 128 ** 3 + 44 * smp, flops=0)
    if kind == "multi":
        n = sum(_multi_rays(case))
        return dict(bytes=n * (24 + 8 + 1 + 9) + case["scenes"] * 128 ** 3 + 44 * MULTI_MEAN * n, flops=0)
    if kind == "volume":
        S, R = case["samples"], case["samples"] / case["mean"]
        # sigma, rgb, dt, m, dt_norm in; d sigma, d rgb out; rgba, dist and their gradients
        return dict(bytes=S * (28 + 16) + R * (8 + 20 + 20), flops=60 * S)
    if kind == "losses":
        S, R = case["samples"], case["samples"] / case["mean"]
        return dict(bytes=S * (32 + 16) + R * (8 + 28 + 16), flops=60 * S)
    if kind == "occupancy":
        V = case["resolution"] ** 3
        return dict(bytes=8 * case["cascades"] * V + V + case["updates"] * (4 + 4 + 12 + 12 + 8), flops=0)
    if kind == "adam":
        n = case["grid"] + case["mlp"]
        return dict(bytes=4 * n + 32 * (case["grid"] * case["touched"] + case["mlp"]), flops=15 * n)
    if kind == "hashgrid":
        n, f = case["samples"], 2 * case["levels"]
        table = min(8 << case["log2_table"], 64 * n) * case["levels"]
        # positions, features out and their gradients in; the touched entries read, the gradients written
        return dict(bytes=n * (12 + 8 * f) + table + (8 << case["log2_table"]) * case["levels"], flops=40 * n * f)
    if kind in ("trainer", "image_trainer"):
        b, V = case["batch"], 128 ** 3
        # rays, emitted samples, losses, Adam over the touched half, the occupancy update
        total = case["rays"] * 41 + 40 * b + 48 * b + 16 * (1 << 20) * (4 + 16) + 41 * V + 48 * case["updates"]
        if kind == "image_trainer":
            total += b * 32 * 16 + 2 * (64 << 20)
        return dict(bytes=total, flops=100 * b)
    if kind == "render":
        px = case["width"] * case["height"]
        return dict(bytes=16 * px + 128 ** 3, flops=2000 * px)
    raise ValueError(kind)


# ---- outputs in 64 bits ----------------------------------------------------------------------
def _seg_excl(x, off, ray):
    """Exclusive running sum of x inside each ray."""
    e = torch.cumsum(x, 0) - x
    return e - e[off.clamp_max(x.numel() - 1)][ray]


def _seg_total(x, R, ray):
    return torch.zeros(R, dtype=torch.float64, device=DEV).index_add_(0, ray, x)


def _sigma64(b, activation):
    d = b["density"].detach().double()
    return (d, torch.ones_like(d)) if activation == 0 else (torch.exp(d.clamp(max=12.0) - 1.0),) * 2


def _composite64(b, activation, min_t=1e-4):
    off, ray, R = b["offsets"].long(), b["ray"], b["counts"].numel()
    sig, dsig = _sigma64(b, activation)
    dt, rgb = b["dt"].double(), b["rgb"].detach().double()
    x = sig * dt
    X = _seg_excl(x, off, ray)
    first = torch.zeros_like(ray, dtype=torch.bool)
    first[off[b["counts"] > 0]] = True
    live = (torch.exp(-X) >= min_t) | first
    w = torch.exp(-X) * -torch.expm1(-x) * live
    rgba = torch.stack([_seg_total(w * rgb[c], R, ray) for c in range(3)] + [_seg_total(w, R, ray)])
    return dict(rgba=rgba, w=w, live=live, after=torch.exp(-(X + x)), rgb=rgb, dt=dt, dsig=dsig, off=off, ray=ray, R=R)


def _composite_vjp64(c, g):
    """d sigma (through the activation) and d rgb for the upstream g [4][R]."""
    gr = g[:, c["ray"]]
    u = (gr[:3] * c["rgb"]).sum(0) + gr[3]
    wu = c["w"] * u
    after = _seg_total(wu, c["R"], c["ray"])[c["ray"]] - _seg_excl(wu, c["off"], c["ray"]) - wu
    return c["dt"] * (c["after"] * u - after) * c["dsig"] * c["live"], gr[:3] * c["w"]


def _distortion64(b, activation, lam):
    off, ray, R = b["offsets"].long(), b["ray"], b["counts"].numel()
    sig, dsig = _sigma64(b, activation)
    dtn, m = b["dt_norm"].double(), b["m_norm"].double()
    x = sig * dtn
    X = _seg_excl(x, off, ray)
    w = torch.exp(-X) * -torch.expm1(-x)
    W, WM = _seg_excl(w, off, ray), _seg_excl(w * m, off, ray)
    A = m * W - WM
    k = lam / b["counts"].double()[ray]
    loss = _seg_total(k * (dtn * w * w / 3.0 + 2.0 * w * A), R, ray)
    B = (_seg_total(w * m, R, ray)[ray] - WM - w * m) - m * (_seg_total(w, R, ray)[ray] - W - w)
    dw = k * (2.0 / 3.0 * dtn * w + 2.0 * (A + B))
    dww = dw * w
    after = _seg_total(dww, R, ray)[ray] - _seg_excl(dww, off, ray) - dww
    return loss, dtn * (dw * torch.exp(-(X + x)) - after) * dsig


def _exact_losses(case, seed):
    b = _batch(seed, case["samples"], case["mean"], case["activation"])
    c = _composite64(b, case["activation"])
    R = c["R"]
    R_, a = c["rgba"][:3], c["rgba"][3]
    tgt, bg = b["target"].double(), b["bg"].double()
    gt = tgt[:3] * tgt[3] + bg * (1.0 - tgt[3])
    pred = R_ * a + bg * (1.0 - a)
    d = torch.cat([pred - gt, ((1.0 - a) - (1.0 - tgt[3]))[None]])
    ad = d.abs()
    loss = torch.where(ad < 1.0, 0.5 * d * d, ad - 0.5).sum() / R
    up = torch.where(ad < 1.0, d, torch.sign(d))[:3] / R
    g = torch.cat([up * a, (up * (R_ - bg)).sum(0, keepdim=True)])
    rec, d_rgb = _composite_vjp64(c, g)
    dl, dist = _distortion64(b, case["activation"], LAMBDA)
    t = b["t"].double()
    grad = (rec + dist) * torch.where(t < 1.0, t * t, torch.ones_like(t))
    return dict(rgba=c["rgba"].view(-1), grad=grad, d_rgb=d_rgb.reshape(-1), sums=torch.stack([loss, dl.mean()]))


def _exact_volume(case, seed):
    b = _batch(seed, case["samples"], case["mean"], case["activation"])
    c = _composite64(b, case["activation"])
    ds, d_rgb = _composite_vjp64(c, b["grad_rgba"].double())
    dl, dd = _distortion64(b, case["activation"], LAMBDA)
    return dict(rgba=c["rgba"], dist=dl, d_sigma=ds + dd * b["grad_dist"].double()[c["ray"]], d_rgb=d_rgb)


def _exact_adam(case, seed):
    s = _adam_state(case, seed)
    w, g = s["w"].double(), s["g"].double()
    act = g != 0
    act[s["ng"]:] = True
    g[s["ng"]:] += 1e-6 * w[s["ng"]:]
    m, v = 0.1 * g, 0.01 * g * g
    nw = w - 1e-2 * math.sqrt(1 - 0.99) / (1 - 0.9) * m / (v.sqrt() + 1e-15)
    return dict(w=torch.where(act, nw, w), m=m, v=v, steps=None)


def _exact_hashgrid(case, seed):
    s = _hashgrid_state(case, seed)
    spec, n, T = s["spec"], s["n"], 1 << case["log2_table"]
    pos = s["pos"].view(3, n).double()
    P, df = s["params"].double().view(spec.n_levels, T, 2), s["dfeat"].double().view(spec.n_levels, 2, n)
    feat = torch.zeros((spec.n_levels, 2, n), dtype=torch.float64, device=DEV)
    grads = torch.zeros((spec.n_levels, T, 2), dtype=torch.float64, device=DEV)
    for l in range(spec.n_levels):
        res, dense = spec.level(l)
        x = (pos * res).float().double()  # the cell coordinate is an FP32 number by definition
        i = x.floor().clamp(0, res - 1)
        f, i = x - i, i.long()
        for k in range(8):
            bit = [(k >> a) & 1 for a in range(3)]
            wt = torch.ones(n, dtype=torch.float64, device=DEV)
            for a in range(3):
                wt = wt * (f[a] if bit[a] else 1.0 - f[a])
            vx, vy, vz = (i[a] + bit[a] for a in range(3))
            if dense:
                e = vx + (res + 1) * (vy + (res + 1) * vz)
            else:
                e = (vx ^ (vy * 2654435761) ^ (vz * 805459861)) & (T - 1)
            feat[l] += wt * P[l][e].t()
            grads[l].index_add_(0, e, (wt * df[l]).t())
    return dict(feat=feat.view(-1), grads=grads.view(-1))


def _exact_occupancy(case, seed):
    s = _occupancy_state(case, seed)
    R, L, n = case["resolution"], case["cascades"], case["updates"]
    lv, cell = s["levels"].long(), s["cells"].long()
    occ = (s["bits"][cell].long() >> lv) & 1
    sel = torch.ones_like(occ, dtype=torch.bool) if case["all"] else (s["select"] < 0.25) | (
        (s["select"] <= 0.5) & (occ == 1))
    val = torch.exp(s["values"].double().clamp(max=12.0) - 1.0)
    at = lv * R ** 3 + cell
    density = s["density"].double() * 0.95
    density.scatter_reduce_(0, at[sel], val[sel], "amax")
    pos = []
    for a in range(3):
        v = cell >> a
        q = torch.zeros_like(v)
        for bit in range(10):
            q |= ((v >> (3 * bit)) & 1) << bit
        vs = (2.0 ** lv.double()) / R
        pos.append(((q - R // 2).double() + s["rand3"][a * n:(a + 1) * n].double()) * vs * s["inv"] + 0.5)
    return dict(pos=torch.cat(pos), density=density, bits=None, count=None)


def exact(case, seed):
    """None for the marches, the whole steps and the render: their outputs are the FP32 recurrence of
    the step positions and what follows from it, which 64 bits would not reproduce."""
    f = dict(volume=_exact_volume, losses=_exact_losses, adam=_exact_adam, hashgrid=_exact_hashgrid,
             occupancy=_exact_occupancy).get(case["kind"])
    return f(case, seed) if f else None
