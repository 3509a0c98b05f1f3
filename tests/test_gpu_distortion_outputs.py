"""The distortion loss's gradient when the loss itself is not asked for: that launch leaves out the
loss sums and the forward of each warp's last tile (128 samples), and its gradient has to be the one
of the launch that makes both, bit for bit."""
import numpy as np
import pytest
import torch

from tests.helpers import assert_bitwise, dev, host, i32

pytestmark = pytest.mark.gpu


def _counts(kind):
    rng = np.random.default_rng(11)
    if kind == "edges":  # rays that end at, before and after a tile's end, and empty ones
        return np.array([1, 127, 128, 129, 0, 255, 256, 257, 0, 3, 383, 385, 1, 0], np.uint32)
    if kind == "short":  # many rays a tile
        return rng.integers(0, 9, 5000).astype(np.uint32)
    if kind == "one":
        return np.array([1], np.uint32)
    return np.array([128 * 64, 128 * 66 + 5, 128 * 65, 7], np.uint32)  # past the kept carries


@pytest.mark.parametrize("activation", [0, 1])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("kind", ["edges", "short", "one", "long"])
def test_gradient_without_the_loss(kind, shift, activation):
    from turbonerf_b200 import hotpath as hp
    counts = _counts(kind)
    n, first = len(counts), 3 * shift
    offsets = (np.cumsum(counts) - counts + first).astype(np.uint32)
    ss = int(counts.sum()) + first
    ss += -ss % 4 if shift == 0 else 0
    rng = np.random.default_rng(3)
    sigma = rng.normal(-1.0, 1.0, ss).astype(np.float32) if activation else rng.exponential(2.0, ss).astype(np.float32)
    m, dt = np.sort(rng.random(ss)).astype(np.float32), rng.uniform(1e-3, 2e-2, ss).astype(np.float32)
    sg, mn, dn = (dev(np.concatenate([np.zeros(shift, np.float32), v]))[shift:] for v in (sigma, m, dt))
    counts_t, offsets_t, grad = i32(counts), i32(offsets), dev(rng.normal(0, 1, n).astype(np.float32))
    ctx = hp.Context()
    rb = hp.ray_batch(counts_t, offsets_t, n, n, ss)
    full = hp.distortion_fwd_bwd(ctx, rb, sg, mn, dn, 0.01, activation=activation, grad_ray=grad)
    dd = torch.full((ss,), 7.0, device="cuda")
    hp.distortion_call(ctx, rb, sg, mn, dn, 0.01, activation, grad, None, None, dd)
    a, b = host(full["dL_ddensity"]), host(dd)
    live = slice(first, first + int(counts.sum()))
    assert_bitwise(a[live], b[live], "gradient")
    assert (b[:first] == 7.0).all() and (b[live.stop:] == 7.0).all(), "samples of no ray are left alone"
    only_loss = torch.zeros(n, device="cuda")
    hp.distortion_call(ctx, rb, sg, mn, dn, 0.01, activation, None, only_loss, None, None)
    assert_bitwise(host(full["ray_loss"]), host(only_loss), "loss")
