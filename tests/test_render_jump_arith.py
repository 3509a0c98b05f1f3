"""Steps of one length taken at once by the render walk's empty-space stretches, in the kernel's
arithmetic on the CPU, against the additions one by one in float32."""
import numpy as np
import pytest

f32 = np.float32


def steps_at_once(t, d, lim, max_steps):
    """(t after n steps, n, stop), as steps_at_once in csrc/render.cu."""
    bits = int(t.view(np.uint32))
    e = bits >> 23
    if not 32 <= e < 232:
        return t, 0, t
    stop = min(lim, np.uint32(bits | 0x7FFFFF).view(f32))
    per_ulp = np.uint32((277 - e) << 23).view(f32)
    with np.errstate(over="ignore"):
        q = f32(d * per_ulp)
        inc = np.rint(q)
        room = f32(f32(stop - t) * per_ulp)
        if not room > f32(8) * inc or not inc >= 1 or abs(f32(q - inc)) == f32(0.5):
            return t, 0, stop
    n = min(int(f32(room / inc)) - 1, max_steps)
    return np.uint32(bits + n * int(inc)).view(f32), n, stop


def stretch(t, d, t_out, cap):
    """The kernel's loop over one stretch of constant steps; also whether any were taken at once."""
    iters, jumped = 0, 0
    while t <= t_out and iters < cap:
        t, n, stop = steps_at_once(t, d, t_out, cap - iters - 1)
        iters, jumped = iters + n, jumped + n
        while True:
            t = f32(t + d)
            iters += 1
            if not (t <= stop and iters < cap):
                break
    return t, iters, jumped


@pytest.mark.parametrize("kind", ["any", "few bits", "tiny", "wide"])
def test_steps_at_once_are_the_single_steps(kind):
    rng = np.random.default_rng(len(kind))
    total = 0
    for case in range(60):
        if kind == "few bits":  # halfway cases: one significant bit of d at half an ulp of t
            d = f32(np.ldexp(float(rng.integers(1, 8)), int(rng.integers(-16, -6))))
            t = f32(np.exp(rng.uniform(np.log(1e-3), np.log(4e5))))
        elif kind == "tiny":  # from zero, and steps near or below the ulp
            d = f32(np.exp(rng.uniform(np.log(1e-8), np.log(1e-6))))
            t = f32(rng.choice([0.0, 1e-30, 0.4, 3.9, 7.99]))
        else:
            d = f32(np.exp(rng.uniform(np.log(1e-4), np.log(2e-2 if kind == "any" else 3.0))))
            t = f32(rng.choice([0.0, rng.uniform(0, 30)]))
        t_out = f32(float(t) + float(d) * rng.uniform(0.0, 3000.0))
        if case % 7 == 0:  # an end on a step, or on a power of two
            t_out = f32(np.exp2(np.ceil(np.log2(max(float(t_out), 1e-6)))))
        cap = int(rng.choice([4000, rng.integers(1, 60)]))
        one, n = t, 0
        while one <= t_out and n < cap:
            one, n = f32(one + d), n + 1
        got, m, jumped = stretch(t, d, t_out, cap)
        assert got == one and m == n, (kind, t, d, t_out, cap)
        total += jumped
    assert total > 1000
