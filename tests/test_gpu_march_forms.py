"""The forms of the march count loop (bitfield bytes, coarse mip, box inside the grid, power-of-two
level sizes) against the CPU oracle, bit for bit, on random bitfields, whose occupancy changes at
almost every step: the lookups that run behind the loop's steps then turn up wrong most often."""
import numpy as np
import pytest

import oracle
from tests.helpers import assert_bitwise, dev, host
from turbonerf_b200 import scenes

pytestmark = pytest.mark.gpu

# resolution, levels, base size, half box size, occupied share, cone, max_steps, max_iterations
CASES = {
    "pow2": (128, 5, 1.0, 8.0, 0.2, 1 / 256, 0, 0),
    "pow2_dense_limit": (32, 3, 0.5, 1.0, 0.7, 1 / 256, 37, 0),
    "any_size": (64, 4, 0.3, 1.2, 0.3, 1 / 256, 0, 0),
    "any_size_fixed_dt": (16, 1, 3.0, 1.5, 0.5, 0.0, 100, 0),
    "box_past_grid": (32, 2, 1.0, 3.0, 0.3, 1 / 256, 0, 0),
    "bytes_small": (8, 3, 1.0, 2.0, 0.4, 1 / 256, 0, 0),
    "bytes_large": (256, 2, 1.0, 1.0, 0.1, 1 / 256, 0, 0),
    "guard": (64, 3, 1.0, 2.0, 0.3, 1 / 256, 0, 25),
    "full": (128, 2, 1.0, 1.0, 1.0, 1 / 256, 0, 0),
    "empty": (128, 2, 1.0, 1.0, 0.0, 1 / 256, 0, 0),
}


@pytest.mark.parametrize("name", CASES)
def test_march_forms(name):
    from turbonerf_b200 import hotpath as hp
    res, levels, base, half, share, cone, max_steps, max_iters = CASES[name]
    rng = np.random.default_rng(list(CASES).index(name))
    bits = np.zeros(res ** 3, np.uint8)
    for k in range(levels):
        bits |= (rng.random(res ** 3) < share).astype(np.uint8) << np.uint8(k)
    n = 333  # a ragged last block
    rays = scenes.sphere_rays(rng, n, radius=2.5 * half, jitter=0.2)
    # rays along the axes, in the faces' planes and from inside
    for i, (o, d) in enumerate([((-2 * half, 0, 0), (1, 0, 0)), ((0, 0, 0), (0, 1, 0)),
                                ((-2 * half, half, half / 4), (1, 0, 0)), ((half / 2, -2 * half, -half), (0, 1, 0)),
                                ((0.1, 0.1, 0.1), (0.6, 0.8, 0.0))]):
        for c in range(3):
            rays.ori[c * n + i], rays.dir[c * n + i] = o[c], d[c]
    box = (-half, -half, -half, half, half, half)
    rays = scenes.rays_init_bbox(rays, box)
    dt = float(scenes.MIN_STEP_SIZE)
    dt_max = float(np.float32(max(2 * half, 1.0)) * np.float32(dt))
    march = dict(bbox=box, cone=cone, dt_min=dt, dt_max=dt_max, max_steps=max_steps)
    grid = dict(n_levels=levels, res=res, base=base, bitfield=bits)
    ns_o, alive_o, _ = oracle.march_count(rays.as_dict(), grid, march, **({"max_iters": max_iters} if max_iters else {}))
    total = int(ns_o.sum())
    off_o = np.zeros(n, np.uint32)
    off_o[1:] = np.cumsum(ns_o[:-1])
    ss = total + 16

    ctx = hp.Context()
    g, m = hp.GridSpec(levels, res, base), hp.MarchSpec(cone, dt, dt_max, max_steps, max_iters)
    ori, dr, t, tmax, alive = dev(rays.ori), dev(rays.dir), dev(rays.t), dev(rays.t_max), dev(rays.alive)
    bits_d = dev(bits)
    ns, info = hp.march_count(ctx, g, bits_d, box, m, n, n, ori, dr, t, tmax, alive, 0xFFFFFFFF)
    assert_bitwise(host(ns).view(np.uint32), ns_o, "n_steps")
    assert_bitwise(host(alive), alive_o, "alive")
    assert int(host(info).view(np.uint32)[1]) == total
    if max_iters or total == 0:
        # some ray runs into the iteration limit; a batch without samples is flagged
        assert ctx.check() != 0
    if total == 0 or max_iters:
        return
    off, smp = hp.march_emit(ctx, g, bits_d, box, m, 0.5 / half, n, n, ss, info, ori, dr, t, alive, ns)
    assert ctx.check() == 0
    em = oracle.march_emit(rays.as_dict(), grid, march, off_o, ns_o, alive_o, n, ss, 0.5 / half)
    assert_bitwise(host(off).view(np.uint32), off_o, "offsets")
    for key in ("t", "dt", "m_norm", "dt_norm"):
        assert_bitwise(host(smp[key])[:total].view(np.uint32), em[key][:total].view(np.uint32), key)


def _few_alive(n, alive_at, rng):
    """n rays of which those at alive_at march through the single-cascade scene."""
    sc = scenes.march_scene_cascaded(n_rays=len(alive_at), n_levels=3)
    r = scenes.RayBatch(n, n, np.zeros(3 * n, np.float32), np.ones(3 * n, np.float32), np.zeros(n, np.float32),
                        np.zeros(n, np.float32), np.zeros(n, np.uint8))
    k = len(alive_at)
    for c in range(3):
        r.ori[c * n + alive_at], r.dir[c * n + alive_at] = sc.rays.ori[c * k:(c + 1) * k], sc.rays.dir[c * k:(c + 1) * k]
    r.t[alive_at], r.t_max[alive_at], r.alive[alive_at] = sc.rays.t, sc.rays.t_max, sc.rays.alive
    return sc, r


@pytest.mark.parametrize("n,rpw", [(4_200_000, 1), (4_200_000, 2), (4_200_000, 4), (300, 1), (300, 4), (5000, 2)])
def test_emit_past_the_slots_and_in_parts(n, rpw):
    """4.2 million rays leave 16 step slots a ray, fewer than the marching rays have samples, so the
    emit pass marches on; a few hundred rays are spread over several warps each."""
    from turbonerf_b200 import hotpath as hp
    rng = np.random.default_rng(n)
    at = np.sort(rng.choice(n, 200, replace=False))
    sc, r = _few_alive(n, at, rng)
    march = dict(bbox=sc.bbox, cone=sc.cone_angle, dt_min=sc.dt_min, dt_max=sc.dt_max, max_steps=0)
    ns_o, alive_o, _ = oracle.march_count(r.as_dict(), sc.grid.as_dict(), march)
    assert ns_o.max() > 64
    off_o = np.concatenate([[0], np.cumsum(ns_o[:-1])]).astype(np.uint32)
    total = int(ns_o.sum())
    em = oracle.march_emit(r.as_dict(), sc.grid.as_dict(), march, off_o, ns_o, alive_o, n, total, 1.0 / sc.aabb_size)
    ctx = hp.Context()
    ctx.tuning = {"emit_rays_per_warp": rpw}
    g, m = hp.GridSpec(3, 128, 1.0), hp.MarchSpec(sc.cone_angle, sc.dt_min, sc.dt_max, 0)
    ori, dr, t, tmax, alive = dev(r.ori), dev(r.dir), dev(r.t), dev(r.t_max), dev(r.alive)
    bits = dev(sc.grid.bitfield)
    ns, info = hp.march_count(ctx, g, bits, sc.bbox, m, n, n, ori, dr, t, tmax, alive, 0xFFFFFFFF)
    off, smp = hp.march_emit(ctx, g, bits, sc.bbox, m, 1.0 / sc.aabb_size, n, n, total, info, ori, dr, t, alive, ns)
    assert ctx.check() == 0
    assert_bitwise(host(ns).view(np.uint32), ns_o, "n_steps")
    assert_bitwise(host(off).view(np.uint32), off_o, "offsets")
    for key in ("t", "pos", "dir", "dt", "m_norm", "dt_norm"):
        assert_bitwise(host(smp[key]).view(np.uint32), em[key].view(np.uint32), key)
    # the same rays as one scene of a multi-scene launch
    table = hp.scene_table([dict(grid=g, bitfield=bits, bbox=sc.bbox, march=m, inv_aabb=1.0 / sc.aabb_size,
                                 ray_begin=0, n_rays=n)])
    alive = dev(r.alive)
    ns2, _, _ = hp.multi_march_count(ctx, table, n, ori, dr, t, tmax, alive)
    off2, smp2 = hp.multi_march_emit(ctx, table, n, total, ori, dr, t, alive, ns2)
    assert ctx.check() == 0
    for key in ("t", "pos", "m_norm"):
        assert_bitwise(host(smp2[key]).view(np.uint32), em[key].view(np.uint32), "multi " + key)
