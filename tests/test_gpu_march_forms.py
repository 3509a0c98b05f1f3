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
