"""The march count around the number of rays that gives every warp scheduler one warp, where it goes from
more steps in flight to fewer: counts against the CPU oracle, bit for bit, on random bitfields."""
import numpy as np
import pytest
import torch

import oracle
from tests.helpers import assert_bitwise, dev, host
from turbonerf_b200 import scenes

pytestmark = pytest.mark.gpu

# resolution, levels, base size, half box size, occupied share
GRIDS = {"pow2": (64, 3, 1.0, 2.0, 0.3), "bounded": (64, 3, 0.3, 0.6, 0.3), "box_past_grid": (32, 2, 1.0, 3.0, 0.1),
         "bytes": (8, 2, 1.0, 1.0, 0.3)}


@pytest.mark.parametrize("past", [0, 1])
@pytest.mark.parametrize("name", GRIDS)
def test_counts_around_one_warp_a_scheduler(name, past):
    from turbonerf_b200 import hotpath as hp
    res, levels, base, half, share = GRIDS[name]
    n = torch.cuda.get_device_properties(0).multi_processor_count * 128 + past
    rng = np.random.default_rng(list(GRIDS).index(name))
    bits = np.zeros(res ** 3, np.uint8)
    for k in range(levels):
        bits |= (rng.random(res ** 3) < share).astype(np.uint8) << np.uint8(k)
    box = (-half,) * 3 + (half,) * 3
    rays = scenes.rays_init_bbox(scenes.sphere_rays(rng, n, radius=2.5 * half, jitter=0.2), box)
    dt = float(scenes.MIN_STEP_SIZE)
    dt_max = float(np.float32(max(2 * half, 1.0)) * np.float32(dt))
    ns_o, alive_o, _ = oracle.march_count(rays.as_dict(), dict(n_levels=levels, res=res, base=base, bitfield=bits),
                                          dict(bbox=box, cone=1 / 256, dt_min=dt, dt_max=dt_max))
    alive = dev(rays.alive)
    ctx = hp.Context()
    ns, _ = hp.march_count(ctx, hp.GridSpec(levels, res, base), dev(bits), box, hp.MarchSpec(1 / 256, dt, dt_max, 0), n, n,
                           dev(rays.ori), dev(rays.dir), dev(rays.t), dev(rays.t_max), alive, 0xFFFFFFFF)
    assert ctx.check() == 0
    assert_bitwise(host(ns).view(np.uint32), ns_o, "n_steps")
    assert_bitwise(host(alive), alive_o, "alive")
