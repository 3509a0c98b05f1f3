"""The hash-grid backward's forms: four or eight samples a thread (by the number of samples times
levels), 16-byte groups or single loads (by alignment and stride), paired or single reductions (by
the gradients' alignment), on positions along rays, where consecutive samples share cells, and a
live count that ends inside a thread's run. FP64 oracle, within 1e-5 of the largest gradient: a
gradient is a sum of up to a few thousand FP32 products added in FP32 in any order (2^-24 each,
relative to partial sums no larger than the sum of magnitudes, which random signs keep within
some tens of the result)."""
import numpy as np
import pytest

import oracle
from tests.helpers import assert_norm_close, dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,live,pad,shift,levels", [
    (70_001, 70_001, 0, 0, 16),      # 8 a thread, odd stride: single loads
    (70_004, 69_997, 0, 0, 16),      # 8 a thread, 16-byte groups, a ragged end
    (70_004, 70_004, 0, 2, 16),      # gradients 8-byte aligned only
    (3000, 2999, 0, 0, 5),           # 4 a thread, 16-byte groups
    (3001, 3001, 6, 0, 5),           # 4 a thread, stride past n
    (5, 5, 3, 0, 2),
])
def test_backward_forms(n, live, pad, shift, levels):
    import torch
    from turbonerf_b200 import hotpath as hp
    spec = hp.HashgridSpec(levels, 14, 16.0, 1.4)
    lv = oracle.hashgrid_levels(levels, 14, 16.0, np.float32(1.4))
    rng = np.random.default_rng(n + shift)
    stride = n + pad
    rays = (n + 31) // 32
    o, d = rng.uniform(0, 1, (rays, 1, 3)), rng.normal(size=(rays, 1, 3))
    d /= np.linalg.norm(d, axis=2, keepdims=True)
    p = np.clip(o + d * np.arange(32)[None, :, None] * 0.002, 0, 1).reshape(-1, 3)[:n]
    pos = np.zeros((3, stride), np.float32)
    pos[:, :n] = p.T
    nf = spec.n_features
    dfeat = np.zeros((nf, stride), np.float32)
    dfeat[:, :live] = rng.normal(size=(nf, live))
    poison = dfeat.copy()
    poison[:, live:] = 1e9  # past the live count: must not be read into a gradient
    n_hash, _ = spec.n_params()
    buf = torch.zeros(n_hash + shift, device="cuda")
    grads = buf[shift:]
    n_dev = torch.tensor([live], dtype=torch.int32, device="cuda")
    hp.hashgrid_backward(spec, dev(pos.ravel()), dev(poison.ravel()), grads, n, stride, n_dev=n_dev, touched=False)
    ref, _ = oracle.hashgrid_backward(lv, 14, np.ascontiguousarray(pos[:, :live]).ravel(),
                                      np.ascontiguousarray(dfeat[:, :live]).ravel().astype(np.float64), live)
    g = host(grads).astype(np.float64)
    T = 1 << 14
    for l in range(levels):
        sl = slice(2 * l * T, 2 * (l + 1) * T)
        assert_norm_close(g[sl], ref[sl], 1e-5, f"level {l} gradients")
