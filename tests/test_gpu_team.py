"""The solver with a team of lanes per particle (scenes of at most 16,384
particles) gives the bits of the one-lane solver: the same scenes in engines of
their own (teams) and together in a batch too large for teams."""
import numpy as np
import pytest

from mtlphys_b200 import Engine, _abi
from mtlphys_b200.batch import Batch
from parity import random_scene

pytestmark = pytest.mark.gpu
LIMIT = 16384


def cloud(seed, n):
    """A random cloud with clumps of hundreds of particles per cell (rows of many
    chunks), or for small n a single tight clump."""
    if n >= 100:
        return random_scene(seed, n)
    rng = np.random.default_rng(seed)
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0.0, 0.15, (n, 3))
    return pos, np.zeros((n, 4), np.float32)


@pytest.mark.parametrize("scorr_n, iterations", [(4, 3), (3, 1), (4, 2)])
def test_team_and_one_lane_solvers_give_the_same_bits(cuda, scorr_n, iterations):
    counts = [1, 2, 33, 700, 4099, LIMIT]
    states = [cloud(s, n) for s, n in enumerate(counts)]
    p = _abi.default_params()
    p.set(scorr_n=scorr_n, scorr_k=0.01, solver_iterations=iterations)
    dt = 1.0 / 120.0
    which = (_abi.MP_BUF_POSITIONS, _abi.MP_BUF_VELOCITIES, _abi.MP_BUF_LAMBDAS, _abi.MP_BUF_FOAM,
             _abi.MP_BUF_NEIGHBOR_COUNTS)
    b = Batch(0)
    try:
        b.reset(counts, p, [dt] * len(counts))
        assert b.particle_count() > LIMIT
        b.write(_abi.MP_BUF_POSITIONS, np.concatenate([x for x, _ in states]))
        b.write(_abi.MP_BUF_VELOCITIES, np.concatenate([v for _, v in states]))
        for _ in range(2):
            b.step()
        assert b.check_errors() == 0
        together = [b.read(w) for w in which]
        ranges = [b.scene_range(s) for s in range(len(counts))]
    finally:
        b.close()
    for (first, n), (pos, vel) in zip(ranges, states):
        e = Engine(0)
        try:
            e.set_params(p)
            e.reset(n, _abi.MP_SCENE_CUBE_DROP)
            e.set_positions(pos)
            e.set_velocities(vel)
            for _ in range(2):
                e.step(dt)
            assert e.check_errors() == 0
            for w, all_scenes in zip(which, together):
                np.testing.assert_array_equal(e.read(w), all_scenes[first:first + n], err_msg=f"{n} particles, buffer {w}")
        finally:
            e.close()
