"""The render walk's steps of constant length taken at once, at step sizes of few significant bits
(whose multiples fall halfway between floats at some t), ordinary ones, small and large ones:
the samples of every ray have to be the step-by-step ones."""
import numpy as np
import pytest

from tests.test_gpu_render import _camera, _compare, _oracle_image, _submit, _trainer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt_min", [2.0 ** -10, 1.5 * 2.0 ** -11, 5.0 * 2.0 ** -12, 1.7e-3, 3.1e-4, 2.3e-2])
def test_steps_at_once_give_the_same_samples(dt_min):
    rng = np.random.default_rng(7)
    bits = np.zeros(128 ** 3, np.uint8)
    for k in range(5):
        bits |= ((rng.random(128 ** 3) < 4e-4).astype(np.uint8) << np.uint8(k))
    sc, tr = _trainer(min_transmittance=0.0, bitfield=bits)
    for eye in ((0.3, 0.8, 4.0), (0.05, -0.2, 0.3), (12.0, 3.0, -9.0)):
        cam = _camera(24, 20, eye)
        img, stats = _submit(tr, cam, batch_size=1 << 16, min_step_size=dt_min)
        ref, amb, n_ref = _oracle_image(sc, cam, dt_min=dt_min, min_t=0.0)
        assert stats["samples"] == n_ref, (eye, stats, n_ref)
        _compare(img, ref, amb, f"dt_min {dt_min} eye {eye}")
    tr.teardown()
