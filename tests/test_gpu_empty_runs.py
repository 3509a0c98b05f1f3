"""Long runs of rays without samples (an image's background) beside rays with some: the distortion and
compositor launches share such a run between their warps. Values against the CPU oracle, every ray
written; and the launch does not take longer by more than the run's share of the work."""
import numpy as np
import pytest
import torch

import oracle
from tests.helpers import RTOL_COMPOSITE, RTOL_GRAD, assert_close, assert_per_ray_norm_close, dev, host, i32

pytestmark = pytest.mark.gpu


def _counts(where, n_live, n_empty, rng):
    live, none = rng.integers(1, 60, n_live), np.zeros(n_empty, np.int64)
    half = n_live // 2
    return np.concatenate(dict(start=[none, live], middle=[live[:half], none, live[half:]], end=[live, none],
                               all=[none])[where]).astype(np.uint32)


def _batch(counts, rng):
    ss = max(int(counts.sum()), 4)
    ss += -ss % 4
    sigma, dt = rng.exponential(2.0, ss).astype(np.float32), rng.uniform(1e-3, 3e-3, ss).astype(np.float32)
    return dict(ss=ss, off=(np.cumsum(counts) - counts).astype(np.uint32), sigma=sigma, dt=dt,
                rgb=rng.random(3 * ss).astype(np.float32), m=np.sort(rng.random(ss)).astype(np.float32))


@pytest.mark.parametrize("n_live,n_empty", [(40, 300), (700, 33), (9000, 70000)])
@pytest.mark.parametrize("where", ["start", "middle", "end", "all"])
def test_values_beside_runs_of_empty_rays(where, n_live, n_empty):
    from turbonerf_b200 import hotpath as hp
    rng = np.random.default_rng(n_live)
    counts = _counts(where, n_live, n_empty, rng)
    b, n = _batch(counts, rng), len(counts)
    ss, total = b["ss"], int(counts.sum())
    ctx, c, o = hp.Context(), i32(counts), i32(b["off"])
    rb = hp.ray_batch(c, o, n, n, ss)
    sg, dt, rgb, m = dev(b["sigma"]), dev(b["dt"]), dev(b["rgb"]), dev(b["m"])
    nan = lambda k: torch.full((k,), float("nan"), device="cuda")  # noqa: E731
    loss, dd = nan(n), nan(ss)
    hp.distortion_call(ctx, rb, sg, m, dt, 0.01, 0, None, loss, None, dd)
    loss_o, dd_o = oracle.distortion_fwd_bwd(counts, b["off"], b["sigma"], b["m"], b["dt"], 0.01, ss)
    assert_close(host(loss), loss_o, RTOL_GRAD, "distortion loss")
    assert (host(loss)[counts == 0] == 0.0).all()
    assert_close(host(dd)[:total], dd_o[:total], RTOL_GRAD, "distortion gradient")
    out = dict(rgba=nan(4 * n), depth=nan(n), n_used=nan(n).view(torch.int32))
    hp.composite_fwd(ctx, rb, sg, rgb, dt, out=out)
    rgba_o, used_o = oracle.composite_fwd(counts, b["off"], b["sigma"], b["rgb"], b["dt"], n, ss)
    assert_close(host(out["rgba"]), rgba_o, RTOL_COMPOSITE, "rgba")
    assert (host(out["n_used"]).view(np.uint32) == used_o).all()
    grad = rng.normal(0, 1, 4 * n).astype(np.float32)
    cd, crgb = hp.composite_bwd(ctx, rb, sg, rgb, dt, out["depth"], out["n_used"], dev(grad))
    cd_o, crgb_o = oracle.composite_vjp(counts, b["off"], b["sigma"], b["rgb"], b["dt"], grad, n, ss)
    # a gradient in sigma is a difference of larger terms: by rays, as everywhere
    assert_per_ray_norm_close(host(cd), cd_o, counts, b["off"], RTOL_GRAD, "compositor dL/dsigma")
    for k in range(3):
        assert_close(host(crgb)[k * ss:k * ss + total], crgb_o[k * ss:k * ss + total], RTOL_GRAD, "compositor dL/drgb")


def _time(fn):
    fn()
    best = float("inf")
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(5):
            fn()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


def test_time_beside_a_run_of_empty_rays():
    """200,000 empty rays between 9000 others: a warp that took them all needed 100 times as long
    as the batch without them; shared, they take less than the batch does. The line is ten times."""
    from turbonerf_b200 import hotpath as hp
    times = {}
    for n_empty in (0, 200000):
        rng = np.random.default_rng(5)
        counts = _counts("middle", 9000, n_empty, rng)
        b, n = _batch(counts, rng), len(counts)
        ctx, c, o = hp.Context(), i32(counts), i32(b["off"])
        rb = hp.ray_batch(c, o, n, n, b["ss"])
        sg, dt, rgb, m = dev(b["sigma"]), dev(b["dt"]), dev(b["rgb"]), dev(b["m"])
        loss, dd, drgb = (torch.empty(k, device="cuda") for k in (n, b["ss"], 3 * b["ss"]))
        out, grad = hp.composite_fwd(ctx, rb, sg, rgb, dt), torch.ones(4 * n, device="cuda")
        times[n_empty] = [_time(lambda: hp.distortion_call(ctx, rb, sg, m, dt, 0.01, 0, None, loss, None, dd)),
                          _time(lambda: hp.composite_fwd(ctx, rb, sg, rgb, dt, out=out)),
                          _time(lambda: hp.composite_bwd(ctx, rb, sg, rgb, dt, out["depth"], out["n_used"], grad,
                                                         out=(dd, drgb)))]
    for name, with_run, without in zip(("distortion", "compositor", "its gradient"), times[200000], times[0]):
        assert with_run < 10 * without, f"{name}: {with_run:.3f} ms against {without:.3f}"
