"""Bitfields of the resolutions without a coarse mip (below 16, above 128) may start at any byte, a
view into a larger byte tensor: march count and emit, single and multi-scene, against the CPU oracle,
bit for bit."""
import numpy as np
import pytest

import oracle
from tests.helpers import assert_bitwise, dev, host
from turbonerf_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("start", [0, 1, 2, 3])
@pytest.mark.parametrize("res", [2, 8, 256])
def test_bitfield_starts_at_any_byte(res, start):
    import torch
    from turbonerf_b200 import hotpath as hp
    levels, half, n = 2, 1.0, 333
    rng = np.random.default_rng(res + start)
    bits = rng.integers(0, 1 << levels, res ** 3, dtype=np.uint8)
    whole = torch.full((res ** 3 + 8,), 0xFF, dtype=torch.uint8, device="cuda")
    whole[start:start + res ** 3] = dev(bits)
    view = whole[start:start + res ** 3]
    assert view.data_ptr() % 4 == start
    box = (-half,) * 3 + (half,) * 3
    rays = scenes.rays_init_bbox(scenes.sphere_rays(rng, n, radius=2.5, jitter=0.2), box)
    dt, dt_max = float(scenes.MIN_STEP_SIZE), float(np.float32(2 * half) * np.float32(scenes.MIN_STEP_SIZE))
    march = dict(bbox=box, cone=1 / 256, dt_min=dt, dt_max=dt_max)
    grid = dict(n_levels=levels, res=res, base=1.0, bitfield=bits)
    ns_o, alive_o, _ = oracle.march_count(rays.as_dict(), grid, march)
    off_o = np.concatenate([[0], np.cumsum(ns_o[:-1])]).astype(np.uint32)
    total = int(ns_o.sum())
    em = oracle.march_emit(rays.as_dict(), grid, march, off_o, ns_o, alive_o, n, total, 0.5 / half)
    g, m = hp.GridSpec(levels, res, 1.0), hp.MarchSpec(1 / 256, dt, dt_max, 0)
    ori, dr, t, tmax = dev(rays.ori), dev(rays.dir), dev(rays.t), dev(rays.t_max)
    table = hp.scene_table([dict(grid=g, bitfield=view, bbox=box, march=m, inv_aabb=0.5 / half, ray_begin=0, n_rays=n)])
    for multi in (False, True):
        ctx = hp.Context()
        alive = dev(rays.alive)
        if multi:
            ns, _, _ = hp.multi_march_count(ctx, table, n, ori, dr, t, tmax, alive)
            _, smp = hp.multi_march_emit(ctx, table, n, total, ori, dr, t, alive, ns)
        else:
            ns, info = hp.march_count(ctx, g, view, box, m, n, n, ori, dr, t, tmax, alive, 0xFFFFFFFF)
            _, smp = hp.march_emit(ctx, g, view, box, m, 0.5 / half, n, n, total, info, ori, dr, t, alive, ns)
        assert ctx.check() == 0
        assert_bitwise(host(ns).view(np.uint32), ns_o, "n_steps")
        assert_bitwise(host(alive), alive_o, "alive")
        for key in ("t", "dt", "m_norm", "dt_norm"):
            assert_bitwise(host(smp[key]).view(np.uint32), em[key].view(np.uint32), key)
