"""The adjoint's pair sweeps with a team of lanes per slot (at most 16,384
particles) and with one lane per slot give the same gradients: scenes alone in
a batch each, and together in a batch too large for teams."""
import numpy as np
import pytest

from mtlphys_b200 import _abi
from mtlphys_b200.batch import Batch
from parity import random_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scorr_n, iterations", [(4, 3), (3, 1), (0, 2)])
def test_team_and_one_lane_adjoints_agree(cuda, scorr_n, iterations):
    torch = pytest.importorskip("torch")
    counts = [1, 31, 900, 4001, 12400]
    states = [random_scene(s, max(n, 10)) for s, n in enumerate(counts)]
    states = [(x[:n], v[:n]) for (x, v), n in zip(states, counts)]
    grads = [np.random.default_rng(s).normal(size=(n, 4)).astype(np.float32) for s, n in enumerate(counts)]
    p = _abi.default_params()
    p.set(scorr_n=scorr_n, scorr_k=1e-3, epsilon=1e4, solver_iterations=iterations)
    dt = 1.0 / 240.0

    def run(idx):
        b = Batch(0)
        try:
            b.reset([counts[i] for i in idx], p, [dt] * len(idx))
            b.write(_abi.MP_BUF_POSITIONS, np.concatenate([states[i][0] for i in idx]))
            b.write(_abi.MP_BUF_VELOCITIES, np.concatenate([states[i][1] for i in idx]))
            b.rollout_forward(3, 2)
            g = torch.from_numpy(np.concatenate([grads[i] for i in idx])).cuda()
            dp, dv, ds = b.rollout_backward(g, g)
            assert b.check_errors() == 0
            return dp.cpu().numpy(), dv.cpu().numpy(), ds.cpu().numpy()
        finally:
            b.close()

    everyone = run(list(range(len(counts))))
    first = 0
    for i, n in enumerate(counts):
        dp, dv, ds = run([i])
        # the same operations in the same order
        for got, want in zip((dp, dv), everyone[:2]):
            np.testing.assert_array_equal(got, want[first:first + n], err_msg=f"{n} particles")
        np.testing.assert_allclose(ds[0], everyone[2][i], rtol=1e-12, atol=1e-300)  # FP64 sums of the same terms
        first += n
