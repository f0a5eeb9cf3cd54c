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
