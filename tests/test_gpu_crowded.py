"""States that the pair queue and the prefilter were not made for: clumps of
thousands of particles within a few cells, particles far outside the box, hashes
with particles outside their cells.  Results are those of the team kernels or the
oracle; times, against a state of the same kind on another path, stay within
bounds that lie well between what these states cost and what they cost when every
lane walked its queue by itself or every candidate went through it."""
import numpy as np
import pytest

from mtlphys_b200 import Engine, _abi, configs
from mtlphys_b200.batch import Batch
from parity import assert_equal_u32, random_scene

pytestmark = pytest.mark.gpu
DT = 1.0 / 120.0


def cloud_params():
    p = _abi.default_params()
    return p.set(scorr_k=1e-4, solver_iterations=3)


def cube(n, offset=0.0):
    side = int(np.ceil(round(n ** (1.0 / 3.0), 9)))
    i = np.arange(n)
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = 2.0 + 0.05 * np.stack([i % side, i // side ** 2, (i // side) % side], 1)
    pos[:, :3] += np.random.default_rng(1).uniform(-0.005, 0.005, (n, 3))
    pos[:, 0] += offset
    return pos, np.zeros((n, 4), np.float32)


def best_ms(params, pos, vel, hash_only=False, reps=6):
    """Fastest of `reps` passes from one state, in ms."""
    import torch

    e = Engine(0)
    try:
        e.set_params(params)
        e.reset(len(pos), _abi.MP_SCENE_CUBE_DROP)
        state = [(e.tensor(w), torch.from_numpy(x).cuda())
                 for w, x in ((_abi.MP_BUF_POSITIONS, pos), (_abi.MP_BUF_VELOCITIES, vel))]
        times = []
        for _ in range(reps):
            for view, x in state:
                view.copy_(x)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            if hash_only:
                e.build_spatial_hash(torch.cuda.current_stream())
            else:
                e.step(DT, torch.cuda.current_stream())
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)
    finally:
        e.close()


def test_a_warp_walks_full_queues_together(cuda):
    """50,000 particles with clumps of thousands (one lane each) against 16,000 (teams):
    14 times as long; 34 when each lane walked its full queue while the others waited."""
    crowded = best_ms(cloud_params(), *random_scene(3, 50000))
    teams = best_ms(cloud_params(), *random_scene(3, 16000))
    assert crowded < 22.0 * teams, (crowded, teams)


def test_far_particles_test_candidates_exactly_at_once(cuda):
    """100,000 particles 300 m outside the box, where the prefilter cannot place them
    and the border cells hold 184 candidates a row: 12 times an ordinary state; 37 when
    all of them went through the queue."""
    p = configs.base_params(3)
    far, near = best_ms(p, *cube(100000, 300.0)), best_ms(p, *cube(100000))
    assert far < 22.0 * near, (far, near)


def test_far_particles_get_the_same_bits_from_teams_and_one_lane(cuda):
    counts = [33, 4001, 16384]
    p = configs.base_params(3)
    p.set(bounds_max=(3.0, 3.0, 3.0))
    states = [cube(n, off) for n, off in zip(counts, (300.0, 41.0, -2000.0))]
    states[1][0][::7, 0] -= 41.0  # far and near ones in one warp
    which = (_abi.MP_BUF_POSITIONS, _abi.MP_BUF_VELOCITIES, _abi.MP_BUF_LAMBDAS, _abi.MP_BUF_NEIGHBOR_COUNTS)
    b = Batch(0)
    try:
        b.reset(counts, p, [DT] * len(counts))
        b.write(_abi.MP_BUF_POSITIONS, np.concatenate([x for x, _ in states]))
        b.write(_abi.MP_BUF_VELOCITIES, np.concatenate([v for _, v in states]))
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
            e.step(DT)
            assert e.check_errors() == 0
            for w, every in zip(which, together):
                np.testing.assert_array_equal(e.read(w), every[first:first + n], err_msg=f"{n} particles, buffer {w}")
        finally:
            e.close()
