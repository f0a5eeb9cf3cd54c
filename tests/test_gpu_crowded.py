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
    and the border cells hold 184 candidates a row: 14 times an ordinary state; 37 when
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


def test_counts_of_crowded_cells_with_strays_go_straight_through(cuda):
    """buildSpatialHash of a crowded cloud with a tenth of its particles outside the
    box, where no inner threshold holds, against the same inside: 1.6 times as long;
    5 times when every candidate went through the queue."""
    pos, vel = random_scene(3, 50000)
    inside = pos.copy()
    inside[:, :3] = np.clip(inside[:, :3], [-2.9, -2.9, -2.9], [2.9, 5.9, 2.9])
    strays = best_ms(cloud_params(), pos, vel, hash_only=True)
    none = best_ms(cloud_params(), inside, vel, hash_only=True)
    assert strays < 3.0 * none, (strays, none)


@pytest.mark.parametrize("n, clump, offset", [(6001, 4000, 0.0), (6001, 300, 0.0), (5000, 0, 300.0), (70, 40, 0.0)])
def test_counts_without_the_inner_threshold_match_the_oracle(cuda, n, clump, offset):
    """Rows of few, dozens and hundreds of candidates, most of them in range or none."""
    from oracle import oracle as O

    rng = np.random.default_rng(6)
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0.0, 1.0, (n, 3))
    pos[:clump, :3] = 0.5 + rng.normal(0, 0.02, (clump, 3))
    pos[:, 0] += np.float32(offset)
    pos[-20:, :3] = rng.uniform(-0.8, 1.8, (20, 3))
    p = _abi.default_params()
    p.set(cell_size=0.1, bounds_min=(0.0,) * 3, bounds_max=(1.0,) * 3)
    e = Engine(0)
    try:
        e.set_params(p)
        e.reset(n, _abi.MP_SCENE_CUBE_DROP)
        e.set_positions(pos)
        e.build_spatial_hash()
        got = e.neighbor_counts()
        assert e.check_errors() == 0
    finally:
        e.close()
    assert_equal_u32(got, O.build_spatial_hash(p, pos)[3], "neighbor counts")
