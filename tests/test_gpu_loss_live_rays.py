"""The fused losses with the live rays known on the device alone: rays that several warps share, short and
empty ones among them, mean samples a ray on both sides of the line between the two ray numberings (128).
Bit for bit what the same live rays give as a batch of their own; nothing past them is written."""
import numpy as np
import pytest
import torch

from tests.helpers import assert_bitwise, dev, host, i32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [4, 8])
@pytest.mark.parametrize("live", [1, 37, 2000, 2999, 3000])
@pytest.mark.parametrize("short", [0.9, 0.3])
def test_live_rays_on_the_device(short, live, w):
    from turbonerf_b200 import hotpath as hp
    rng = np.random.default_rng(live)
    n = 3000
    counts = np.where(rng.random(n) < short, rng.integers(0, 60, n), rng.integers(200, 1100, n)).astype(np.uint32)
    counts[0] = 700
    offsets = (np.cumsum(counts) - counts).astype(np.uint32)
    ss = int(counts.sum())
    ss += -ss % 4
    mean = counts.sum() / n
    assert (mean < 128) == (short == 0.9)
    f = lambda lo, hi, k: dev(rng.uniform(lo, hi, k).astype(np.float32))  # noqa: E731
    args = (f(0, 20, ss), f(0, 1, 3 * ss), f(5e-4, 3e-3, ss), dev(np.sort(rng.random(ss)).astype(np.float32)),
            f(1e-3, 2e-2, ss), f(0, 4, ss), f(0, 1, 4 * n), f(0, 1, 3 * n))
    ctx = hp.Context()
    ctx.tuning = {"loss_rays_per_block": w}
    c, o = i32(counts), i32(offsets)
    end = int(offsets[live - 1] + counts[live - 1])
    out = []
    for rb in (hp.ray_batch(c, o, n, n, ss, i32([live])), hp.ray_batch(c, o, live, n, ss)):
        gd, drgb, rgba, sums = (torch.full((k,), 7.0, device="cuda") for k in (ss, 3 * ss, 4 * n, 2))
        gd[:end] = 0.0
        hp.train_losses(ctx, rb, *args[:6], args[6], args[7], gd, inv_nrays=1.0 / live, lam=1e-3, ray_rgba=rgba,
                        dL_drgb=drgb, loss_sums=sums)
        out.append([host(v) for v in (gd, drgb, rgba)] + [host(sums)])
    for a, b, what in zip(out[0], out[1], ("gradient", "dL/drgb", "rgba")):
        assert_bitwise(a, b, what)
    # the same per-ray terms, added by other threads: each sum of up to 3000 float32 terms
    assert np.allclose(out[0][3], out[1][3], rtol=3000 * 2.0 ** -24, atol=0)
    assert (out[0][0][end:] == 7.0).all() and (out[0][2].reshape(4, n)[:, live:] == 7.0).all()
