"""Scenes of different resolutions in one launch, with and without a coarse mip: counts, offsets and
samples of every scene against the CPU oracle, bit for bit."""
import numpy as np
import pytest

import oracle
from tests.helpers import assert_bitwise, dev, host
from turbonerf_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("resolutions", [(8, 128), (256, 8, 2), (128, 4, 16, 256, 8), (64, 32)])
def test_scenes_of_different_resolutions(resolutions):
    from turbonerf_b200 import hotpath as hp
    levels, half, inv = 2, 1.0, 0.5
    box = (-half,) * 3 + (half,) * 3
    dt, dt_max = float(scenes.MIN_STEP_SIZE), float(np.float32(2 * half) * np.float32(scenes.MIN_STEP_SIZE))
    march = dict(bbox=box, cone=1 / 256, dt_min=dt, dt_max=dt_max)
    table, want, rays, begin = [], [], [], 0
    for k, res in enumerate(resolutions):
        rng = np.random.default_rng(k)
        n = 70 + 41 * k
        bits = ((rng.random(res ** 3) < 0.3) | ((rng.random(res ** 3) < 0.3).astype(np.uint8) << 1)).astype(np.uint8)
        r = scenes.rays_init_bbox(scenes.sphere_rays(rng, n, radius=2.5, jitter=0.2), box)
        grid = dict(n_levels=levels, res=res, base=1.0, bitfield=bits)
        ns, alive, _ = oracle.march_count(r.as_dict(), grid, march)
        off = np.concatenate([[0], np.cumsum(ns[:-1])]).astype(np.uint32)
        em = oracle.march_emit(r.as_dict(), grid, march, off, ns, alive, n, int(ns.sum()), inv)
        table.append(dict(grid=hp.GridSpec(levels, res, 1.0), bitfield=dev(bits), bbox=box,
                          march=hp.MarchSpec(1 / 256, dt, dt_max, 0), inv_aabb=inv, ray_begin=begin, n_rays=n))
        want.append((ns, alive, em))
        rays.append(r)
        begin += n
    R = begin
    join = lambda name, c: np.concatenate([np.concatenate([getattr(r, name).reshape(c, -1)[i] for r in rays])  # noqa: E731
                                           for i in range(c)])
    ori, dr, t, tmax, alive = (dev(join(k, c)) for k, c in (("ori", 3), ("dir", 3), ("t", 1), ("t_max", 1), ("alive", 1)))
    ctx = hp.Context()
    scene_table = hp.scene_table(table)
    ns, per_scene, _ = hp.multi_march_count(ctx, scene_table, R, ori, dr, t, tmax, alive)
    total = sum(int(w[0].sum()) for w in want)
    off, smp = hp.multi_march_emit(ctx, scene_table, R, total, ori, dr, t, alive, ns)
    assert ctx.check() == 0
    ns_o = np.concatenate([w[0] for w in want])
    assert_bitwise(host(ns).view(np.uint32), ns_o, "n_steps")
    assert_bitwise(host(alive), np.concatenate([w[1] for w in want]), "alive")
    assert_bitwise(host(per_scene).view(np.uint32), np.array([w[0].sum() for w in want], np.uint32), "scene samples")
    assert_bitwise(host(off).view(np.uint32), np.concatenate([[0], np.cumsum(ns_o[:-1])]).astype(np.uint32), "offsets")
    for key in ("t", "dt", "m_norm", "dt_norm"):
        assert_bitwise(host(smp[key]).view(np.uint32), np.concatenate([w[2][key] for w in want]).view(np.uint32), key)
