"""Context scratch that is made or grows inside a call on a stream of its own (torch's side streams do not wait for
the legacy default stream): counts and samples equal those of a context reserved beforehand, bit for bit."""
import numpy as np
import pytest
import torch

from tests.helpers import assert_bitwise, dev, host
from turbonerf_b200 import scenes

pytestmark = pytest.mark.gpu


def _march(hp, ctx, rays, n, bits, res, half, total):
    box = (-half,) * 3 + (half,) * 3
    g, m = hp.GridSpec(1, res, 1.0), hp.MarchSpec(0.0, float(scenes.MIN_STEP_SIZE), float(scenes.MIN_STEP_SIZE), 0)
    ori, dr, t, tmax, alive = rays["ori"], rays["dir"], rays["t"], rays["t_max"], rays["alive"].clone()
    ns, info = hp.march_count(ctx, g, bits, box, m, n, n, ori, dr, t, tmax, alive, 0xFFFFFFFF)
    off, smp = hp.march_emit(ctx, g, bits, box, m, 0.5 / half, n, n, total, info, ori, dr, t, alive, ns)
    return ns, off, smp["t"]


@pytest.mark.parametrize("n", [300, 70000])
@pytest.mark.parametrize("res", [128, 8])
@pytest.mark.parametrize("grown", [False, True])
def test_scratch_made_on_a_side_stream(grown, res, n):
    from turbonerf_b200 import hotpath as hp
    half = 0.5
    rng = np.random.default_rng(1)
    r = scenes.rays_init_bbox(scenes.sphere_rays(rng, n, radius=1.5, jitter=0.1), (-half,) * 3 + (half,) * 3)
    rays = {k: dev(getattr(r, k)) for k in ("ori", "dir", "t", "t_max", "alive")}
    # occupied where the rays come in: their first steps are recorded at once
    bits = torch.ones(res ** 3, dtype=torch.uint8, device="cuda")
    total = n * 1100
    total = min(total, 60_000_000)
    ready = hp.Context()
    ready.reserve(n, total)
    want = [host(v).copy() for v in _march(hp, ready, rays, n, bits, res, half, total)]
    small = {k: v.view(-1, n)[:, :64].contiguous().view(-1) for k, v in rays.items()}
    torch.cuda.synchronize()
    for _ in range(5):
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            ctx = hp.Context()
            if grown:  # part of the scratch is there
                _march(hp, ctx, small, 64, bits, res, half, 64 * 1100)
            got = _march(hp, ctx, rays, n, bits, res, half, total)
        torch.cuda.synchronize()
        for g, w, what in zip(got, want, ("n_steps", "offsets", "t")):
            assert_bitwise(host(g), w, what)
