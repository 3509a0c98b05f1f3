"""The distortion launch around the line where it changes from one ray a warp to shares of the samples
(as many rays as a wave of the GPU has warps): values against the CPU oracle, with the live rays known
to the host and on the device alone."""
import numpy as np
import pytest
import torch

import oracle
from tests.helpers import RTOL_GRAD, assert_close, assert_per_ray_norm_close, dev, host, i32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("live", [1.0, 0.6])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("warps_an_sm,off", [(8, 0), (8, 1), (16, 0), (16, 1), (24, -1), (24, 0), (24, 1), (32, 0), (32, 1)])
def test_values_around_one_ray_a_warp(warps_an_sm, off, shift, live):
    from turbonerf_b200 import hotpath as hp
    n = warps_an_sm * torch.cuda.get_device_properties(0).multi_processor_count + off
    rng = np.random.default_rng(n)
    counts = np.where(rng.random(n) < 0.1, 0, rng.integers(1, 40, n)).astype(np.uint32)
    counts[rng.choice(n, 3)] = (128, 700, 128 * 66 + 5)  # past the carries that a warp keeps
    offsets = (np.cumsum(counts) - counts).astype(np.uint32)
    ss = int(counts.sum())
    ss += -ss % 4
    sigma, dt = rng.exponential(0.5, ss).astype(np.float32), rng.uniform(1e-3, 3e-3, ss).astype(np.float32)
    m = np.sort(rng.random(ss)).astype(np.float32)
    sg, mn, dn = (dev(np.concatenate([np.zeros(shift, np.float32), v]))[shift:] for v in (sigma, m, dt))
    k = int(n * live)
    end = int(offsets[k - 1] + counts[k - 1])
    rb = hp.ray_batch(i32(counts), i32(offsets), n, n, ss, None if live == 1.0 else i32([k]))
    loss, dd = torch.full((n,), 7.0, device="cuda"), torch.full((ss,), 7.0, device="cuda")
    grad = rng.normal(0, 1, n).astype(np.float32)
    hp.distortion_call(hp.Context(), rb, sg, mn, dn, 0.01, 0, dev(grad), loss, None, dd)
    loss_o, dd_o = oracle.distortion_fwd_bwd(counts[:k], offsets[:k], sigma, m, dt, 0.01, ss, grad_ray=grad[:k])
    assert_close(host(loss)[:k], loss_o, RTOL_GRAD, "loss")
    assert_per_ray_norm_close(host(dd), dd_o, counts[:k], offsets[:k], RTOL_GRAD, "gradient")
    assert (host(loss)[k:] == 7.0).all() and (host(dd)[end:] == 7.0).all(), "rays past the live ones are left alone"
