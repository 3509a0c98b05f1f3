"""The emit pass of rays with more samples than step slots when the bitfield is no longer the count's:
it ends where the ray leaves the box, or at the iteration limit, and places the samples that it found no
step for there."""
import numpy as np
import pytest

import oracle
from tests.helpers import assert_bitwise, dev, host
from turbonerf_b200 import scenes

pytestmark = pytest.mark.gpu

SLOTS = 1024  # a ray's most
N = 40


@pytest.mark.parametrize("limit", [0, 5])
@pytest.mark.parametrize("multi", [False, True])
@pytest.mark.parametrize("rpw", [1, 4])
def test_bitfield_emptied_before_the_emit(rpw, multi, limit):
    from turbonerf_b200 import hotpath as hp
    half, dt, res = 0.5, float(np.float32(1 / 4096)), 32
    box = (-half,) * 3 + (half,) * 3
    rays = scenes.rays_init_bbox(scenes.sphere_rays(np.random.default_rng(7), N, radius=2.0, jitter=0.05), box)
    bits = np.full(res ** 3, 1, np.uint8)
    march = dict(bbox=box, cone=0.0, dt_min=dt, dt_max=dt)
    ns_o, _, _ = oracle.march_count(rays.as_dict(), dict(n_levels=1, res=res, base=1.0, bitfield=bits), march)
    assert (ns_o > SLOTS + 100).sum() > N // 2
    ctx = hp.Context()
    ctx.tuning = dict(emit_rays_per_warp=rpw)
    g, m, m_emit = hp.GridSpec(1, res, 1.0), hp.MarchSpec(0.0, dt, dt, 0), hp.MarchSpec(0.0, dt, dt, 0, limit)
    ori, dr, t, tmax, alive, bits_d = (dev(a) for a in (rays.ori, rays.dir, rays.t, rays.t_max, rays.alive, bits))
    total = int(ns_o.sum())
    table = lambda spec: hp.scene_table([dict(grid=g, bitfield=bits_d, bbox=box, march=spec, inv_aabb=1.0,  # noqa: E731
                                              ray_begin=0, n_rays=N)])
    if multi:
        ns, _, _ = hp.multi_march_count(ctx, table(m), N, ori, dr, t, tmax, alive)
        bits_d.zero_()
        off, smp = hp.multi_march_emit(ctx, table(m_emit), N, total, ori, dr, t, alive, ns)
    else:
        ns, info = hp.march_count(ctx, g, bits_d, box, m, N, N, ori, dr, t, tmax, alive, 0xFFFFFFFF)
        bits_d.zero_()
        off, smp = hp.march_emit(ctx, g, bits_d, box, m_emit, 1.0, N, N, total, info, ori, dr, t, alive, ns)
    assert ctx.check() == 0
    assert_bitwise(host(ns).view(np.uint32), ns_o, "n_steps")
    off, got = host(off).view(np.uint32), {k: host(smp[k]) for k in ("t", "m_norm", "dt_norm", "dt")}
    f, step = np.float32, np.float32(dt)
    cell = 1.0 / res
    for i in np.nonzero(ns_o > SLOTS)[0]:
        a, b = int(off[i]), int(off[i] + ns_o[i])
        ti, last = got["t"][a:b], got["t"][a + SLOTS - 1]
        assert_bitwise(ti[1:SLOTS], ti[:SLOTS - 1] + step, "recorded positions")
        rest = ti[SLOTS:]
        assert (rest == rest[0]).all()
        p = [f(rays.ori[c * N + i]) + f(rest[0] * rays.dir[c * N + i]) for c in range(3)]
        if limit:
            # a step from the last occupied one, then at most `limit` empty ones, each of at most a cell's diagonal
            assert last + step < rest[0] <= last + step + limit * (1.8 * cell + step)
        else:
            # the first position outside: past the exit by at most one empty step
            assert max(abs(v) for v in p) > half and rest[0] <= rays.t_max[i] + 1.8 * cell + 2 * step
        span = np.maximum(f(f(last + step) - rays.t[i]), f(1e-6))
        mid = (ti + f(0.5) * step).astype(f)
        assert_bitwise(got["m_norm"][a:b], np.clip(((mid - rays.t[i]).astype(f) / span).astype(f), f(0), f(1)), "m_norm")
        assert (got["dt_norm"][a:b] == f(step / span)).all() and (got["dt"][a:b] == step).all()
