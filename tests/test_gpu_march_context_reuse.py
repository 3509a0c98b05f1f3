"""The march count on one context over several grids in turn: nothing of an earlier call's grid may
reach a later call. Counts and alive flags against the CPU oracle, bit for bit; the error word
against a fresh context's, with an iteration limit that only rays cut short where they leave the
occupied cells stay below."""
import numpy as np
import pytest

import oracle
from tests.helpers import assert_bitwise, dev, host
from turbonerf_b200 import scenes

pytestmark = pytest.mark.gpu

N = 333
GUARD = 1  # TN_FLAG_GUARD


def _bits(res, levels, share=0.0, block=None, seed=0):
    """Random occupancy, or (block) the cells lo <= x, y, z < hi of every level alone."""
    rng = np.random.default_rng(seed)
    bits = np.zeros(res ** 3, np.uint8)
    for k in range(levels):
        bits |= (rng.random(res ** 3) < share).astype(np.uint8) << np.uint8(k)
    if block:
        m = np.arange(res ** 3, dtype=np.uint32)
        inside = np.ones(res ** 3, bool)
        for c in range(3):
            x = np.zeros_like(m)
            for b in range(10):
                x |= (m >> np.uint32(3 * b + c) & np.uint32(1)) << np.uint32(b)
            inside &= (x >= block[0]) & (x < block[1])
        bits |= np.where(inside, (1 << levels) - 1, 0).astype(np.uint8)
    return bits


# resolution, levels, half box size, bitfield, iteration limit (0: the default)
STEPS = [
    (128, 1, 0.5, _bits(128, 1, share=1.0), 0),                # fills every block, to the far edges
    (64, 1, 3.0, _bits(64, 1, block=(48, 64)), 0),             # box past the grid, far edge occupied
    (64, 1, 3.0, _bits(64, 1, block=(0, 9)), 0),               # and the near edge
    (8, 3, 2.0, _bits(8, 3, share=0.4, seed=1), 0),            # no coarse mip
    (128, 2, 1.0, _bits(128, 2), 4),                           # nothing occupied: no step is made
    (128, 5, 8.0, _bits(128, 5, share=0.3, seed=2), 0),
    (128, 1, 0.5, _bits(128, 1, block=(58, 70)), 290),         # a few cells in the middle
    (32, 2, 3.0, _bits(32, 2, block=(20, 32)), 0),
]


def _march(ctx, step, rays, box, march):
    from turbonerf_b200 import hotpath as hp
    res, levels, _, bits, limit = step
    alive = dev(rays.alive)
    ns, _ = hp.march_count(ctx, hp.GridSpec(levels, res, 1.0), dev(bits), box,
                           hp.MarchSpec(march["cone"], march["dt_min"], march["dt_max"], 0, limit), N, N, dev(rays.ori),
                           dev(rays.dir), dev(rays.t), dev(rays.t_max), alive, 0xFFFFFFFF)
    return host(ns).view(np.uint32), host(alive), ctx.check()


@pytest.mark.parametrize("group", [32, 256])
def test_grids_in_turn_on_one_context(group):
    from turbonerf_b200 import hotpath as hp
    one = hp.Context()
    one.tuning = dict(count_rays_per_block=group)
    for k, step in enumerate(STEPS):
        res, levels, half, bits, limit = step
        box = (-half,) * 3 + (half,) * 3
        rays = scenes.rays_init_bbox(scenes.sphere_rays(np.random.default_rng(k), N, radius=2.5 * half, jitter=0.2), box)
        dt = float(scenes.MIN_STEP_SIZE)
        march = dict(bbox=box, cone=0.0, dt_min=dt, dt_max=dt)
        grid = dict(n_levels=levels, res=res, base=1.0, bitfield=bits)
        ns_o, alive_o, _ = oracle.march_count(rays.as_dict(), grid, march)
        ns, alive, flags = _march(one, step, rays, box, march)
        assert_bitwise(ns, ns_o, f"step {k}: n_steps")
        assert_bitwise(alive, alive_o, f"step {k}: alive")
        _, _, fresh = _march(hp.Context(), step, rays, box, march)
        assert flags == fresh, f"step {k}: flags {flags:#x}, on a fresh context {fresh:#x}"
        if limit:
            assert not flags & GUARD
            # the limit is one that the whole way through the box exceeds
            assert oracle.march_count(rays.as_dict(), grid, march, limit)[2] > 0
