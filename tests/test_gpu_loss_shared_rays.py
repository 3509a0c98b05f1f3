"""Rays that several warps of the fused loss kernel share (more than 256 and up to 1024 slots, at any
offset in their 16-byte group), among short and empty rays, through the chain of oracle checks of
the fused losses; and the same results for every block size."""
import numpy as np
import pytest

from tests.helpers import assert_bitwise, dev, host, i32
from tests.test_gpu_loss import test_train_losses_fused_matches_oracle_chain as check_chain
from turbonerf_b200 import scenes

pytestmark = pytest.mark.gpu

EDGES = [252, 253, 254, 255, 256, 257, 258, 509, 510, 511, 512, 513, 514, 765, 769, 1020, 1021, 1023, 1024, 1025, 1029]


def _counts(kind):
    rng = np.random.default_rng(5)
    if kind == "edges":
        c = np.repeat(EDGES, 4)
        c = np.concatenate([c, rng.integers(0, 40, 3 * len(c))])  # zero counts among them
    elif kind == "many":  # several shared rays a block and more than one round
        c = rng.integers(1, 700, 1500)
    else:  # a few rays over the whole GPU
        c = np.array([300, 1, 600, 1000])
    rng.shuffle(c)
    return c.astype(np.uint32)


@pytest.mark.parametrize("kind,sigma_scale,shift", [("edges", 1.0, 0), ("edges", 1e-2, 1), ("edges", 1e-3, 0),
                                                    ("many", 1.0, 0), ("few", 1e-2, 0)])
def test_shared_rays_match_oracle(monkeypatch, kind, sigma_scale, shift):
    c = _counts(kind)
    monkeypatch.setattr(scenes, "truncated_geometric_counts", lambda *a, **k: c)
    check_chain(48, 1024, int(c.sum()), sigma_scale, shift)


def test_shared_rays_are_the_same_for_every_block_size(monkeypatch):
    import torch
    from turbonerf_b200 import hotpath as hp
    c = _counts("many")
    monkeypatch.setattr(scenes, "truncated_geometric_counts", lambda *a, **k: c)
    sb = scenes.make_sample_batch(3, int(c.sum()))
    n, ss = sb.n_rays, sb.n_samples
    got = []
    for w in (2, 4, 8):
        ctx = hp.Context()
        ctx.tuning = {"loss_rays_per_block": w}
        counts, offsets = i32(sb.counts), i32(sb.offsets)
        rb = hp.ray_batch(counts, offsets, n, n, ss)
        rgba = torch.zeros(4 * n, device="cuda")
        gd, drgb, _ = hp.train_losses(ctx, rb, dev(sb.sigma), dev(sb.rgb), dev(sb.dt), dev(sb.m_norm), dev(sb.dt_norm),
                                      dev(sb.t), dev(sb.target_rgba), dev(sb.bg_rgb), torch.zeros(ss, device="cuda"),
                                      inv_nrays=1.0 / n, lam=1e-3, ray_rgba=rgba)
        got.append((host(gd), host(drgb), host(rgba)))
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert_bitwise(b, a, "block size")
