"""Gradients in a box so wide that the adjoint compares cells axis by axis are
those of the same particles in a narrow box."""
import numpy as np
import pytest

from mtlphys_b200 import _abi, configs
from mtlphys_b200.batch import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3000, 17000])  # teams, one lane each
def test_wide_and_narrow_boxes_give_the_same_gradients(cuda, n):
    import torch

    rng = np.random.default_rng(11)
    side = int(np.ceil(n ** (1.0 / 3.0)))
    i = np.arange(n)
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = 0.5 + 0.05 * np.stack([i % side, i // side ** 2, (i // side) % side], 1)
    pos[:, :3] += rng.uniform(-0.01, 0.01, (n, 3))
    vel = np.zeros((n, 4), np.float32)
    vel[:, :3] = rng.normal(0.0, 1.0, (n, 3))  # fast enough for one-way pairs
    g = torch.from_numpy(rng.normal(size=(n, 4)).astype(np.float32)).cuda()

    def gradients(width):
        p = configs.base_params(3)
        p.set(scorr_k=1e-3, epsilon=1e4, bounds_max=(width, 3.0, 3.0))
        b = Batch(0)
        try:
            b.reset([n], p, [1.0 / 120.0])
            b.write(_abi.MP_BUF_POSITIONS, pos)
            b.write(_abi.MP_BUF_VELOCITIES, vel)
            b.rollout_forward(3, 2)
            out = [t.cpu().numpy() for t in b.rollout_backward(g, g)]
            assert b.check_errors() == 0
            return [b.positions()] + out
        finally:
            b.close()

    for wide, narrow in zip(gradients(204.75), gradients(8.0)):
        assert np.isfinite(wide).all()
        np.testing.assert_array_equal(wide, narrow)
