"""The compositor's forward into buffers with anything in them: every ray of the batch is written,
those without samples and those whose optical depth is no number too, so the results are the ones
of zeroed buffers, bit for bit."""
import numpy as np
import pytest
import torch

from tests.helpers import assert_bitwise, dev, host, i32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [None, np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("shift", [0, 1])
def test_composite_fwd_writes_every_ray(bad, shift):
    from turbonerf_b200 import hotpath as hp
    rng = np.random.default_rng(2)
    counts = np.concatenate([rng.integers(0, 60, 300), [0, 0, 1, 700, 0]]).astype(np.uint32)
    offsets = (np.cumsum(counts) - counts).astype(np.uint32)
    n, ss = len(counts), int(counts.sum())
    ss += -ss % 4
    sigma, dt = rng.exponential(3.0, ss).astype(np.float32), rng.uniform(1e-3, 3e-2, ss).astype(np.float32)
    rgb = rng.random(3 * ss).astype(np.float32)
    if bad is not None:
        sigma[rng.choice(ss, ss // 40, replace=False)] = bad
    sg, d, col = (dev(np.concatenate([np.zeros(shift, np.float32), v]))[shift:] for v in (sigma, dt, rgb))
    counts_t, offsets_t = i32(counts), i32(offsets)
    ctx = hp.Context()
    rb = hp.ray_batch(counts_t, offsets_t, n, n, ss)
    res = []
    for fill in (0.0, 7.0, float("nan")):
        out = dict(rgba=torch.full((4 * n,), fill, device="cuda"), depth=torch.full((n,), fill, device="cuda"),
                   n_used=torch.full((n,), fill, device="cuda").view(torch.int32))
        res.append(hp.composite_fwd(ctx, rb, sg, col, d, out=out))
    res.append(hp.composite_fwd(ctx, rb, sg, col, d))
    for other in res[1:]:
        for key in ("rgba", "depth", "n_used"):
            assert_bitwise(host(other[key].view(torch.int32)), host(res[0][key].view(torch.int32)), key)
