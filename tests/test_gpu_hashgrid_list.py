"""The hash-grid backward with its list of touched entries, around the line between one launch and two
and at ragged ends of its blocks: along rays, where neighbouring samples share cells, and uniform; single
and paired reductions. List and bits exactly the oracle's; gradients in FP64 within 1e-5 of the largest
of their level (FP32 products added in FP32 in any order)."""
import numpy as np
import pytest

import oracle
from tests.helpers import assert_norm_close, dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["rays", "uniform"])
@pytest.mark.parametrize("n,live,levels,log2_t,shift,pad", [
    (1, 1, 1, 6, 0, 0), (257, 255, 3, 10, 0, 3), (8191, 8191, 16, 12, 2, 0), (8192, 8000, 16, 14, 0, 0),
    (8193, 8193, 16, 14, 0, 1), (26215, 26214, 5, 14, 0, 0), (26214, 26214, 5, 14, 2, 2), (70_001, 512, 4, 15, 0, 0)])
def test_list_forms(n, live, levels, log2_t, shift, pad, how):
    import torch
    from turbonerf_b200 import hotpath as hp
    spec = hp.HashgridSpec(levels, log2_t, 8.0, 1.5)
    lv = oracle.hashgrid_levels(levels, log2_t, 8.0, np.float32(1.5))
    rng = np.random.default_rng(n)
    stride = n + pad
    if how == "rays":
        rays = (n + 31) // 32
        o, d = rng.uniform(0, 1, (rays, 1, 3)), rng.normal(size=(rays, 1, 3))
        d /= np.linalg.norm(d, axis=2, keepdims=True)
        p = np.clip(o + d * np.arange(32)[None, :, None] * 0.002, 0, 1).reshape(-1, 3)[:n]
    else:
        p = rng.random((n, 3))
    pos = np.zeros((3, stride), np.float32)
    pos[:, :n] = p.T
    dfeat = np.full((spec.n_features, stride), 1e9, np.float32)  # past the live count: must not be read into a gradient
    dfeat[:, :live] = rng.normal(size=(spec.n_features, live))
    n_hash, _ = spec.n_params()
    grads = torch.zeros(n_hash + shift, device="cuda")[shift:]
    n_dev = torch.tensor([live], dtype=torch.int32, device="cuda")
    bits, lst, count = hp.hashgrid_backward(spec, dev(pos.ravel()), dev(dfeat.ravel()), grads, n, stride, n_dev=n_dev)
    ref, touched = oracle.hashgrid_backward(lv, log2_t, np.ascontiguousarray(pos[:, :live]).ravel(),
                                            np.ascontiguousarray(dfeat[:, :live]).ravel().astype(np.float64), live)
    k = int(host(count)[0])
    listed = host(lst)[:k].view(np.uint32)
    assert np.array_equal(np.sort(listed), np.nonzero(touched)[0].astype(np.uint32))
    marked = np.unpackbits(host(bits).view(np.uint8), bitorder="little")[:len(touched)]
    assert np.array_equal(marked, (np.asarray(touched) != 0).astype(np.uint8))
    g = host(grads).astype(np.float64)
    for l in range(levels):
        sl = slice(2 * l << log2_t, 2 * (l + 1) << log2_t)
        assert_norm_close(g[sl], ref[sl], 1e-5, f"level {l} gradients")
