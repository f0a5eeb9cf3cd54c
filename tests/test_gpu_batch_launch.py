"""The launch a batch reports is the one its steps use."""
import pytest

from mtlphys_b200 import _abi
from mtlphys_b200.batch import Batch

pytestmark = pytest.mark.gpu


def batch_of(counts, box=None):
    p = _abi.default_params()
    if box:
        p.set(bounds_min=(0.0,) * 3, bounds_max=(box,) * 3)
    b = Batch(0)
    b.reset(counts, p, [1.0 / 120.0] * len(counts))
    return b


@pytest.mark.parametrize("serial", [False, True])
def test_reported_and_tuned_launches_are_what_the_particles_fill(cuda, serial):
    counts = [900, 20000]
    b = batch_of(counts)
    try:
        b.set_serial(serial)
        for block in (128, 256, 512):
            b.set_launch(block)
            # one lane per particle beyond 16,384 particles
            want = -(-(max(counts) if serial else sum(counts)) // block)
            assert b.launch() == (block, want)
            b.set_launch(block, 1)
            assert b.launch()[1] <= want
    finally:
        b.close()


def test_a_tuned_small_batch_does_not_limit_a_larger_one(cuda):
    """Both fall in one bucket of the tuning cache; the small one's grid is the same
    for most block counts per SM, so none of them is a limit."""
    small, large = batch_of([16385]), None
    try:
        assert small.autotune(steps=2)["blocks_per_sm"] >= 1
        block, blocks = small.launch()
        assert blocks == -(-16385 // block)
        large = batch_of([32767])
        assert large.launch() == (block, -(-32767 // block))
    finally:
        small.close()
        if large is not None:
            large.close()


def test_few_particles_in_a_large_box_get_blocks_for_its_cells(cuda):
    """Two particles at opposite corners: the step scans all 4 million cells between
    them, which one block would take milliseconds over: a block per SM.  Near each other,
    the blocks launched for that leave at the first barrier; the results are those of an engine."""
    import numpy as np
    import torch

    from mtlphys_b200 import Engine

    box = 16.0
    b, e = batch_of([2, 3], box), Engine(0)
    try:
        p = b.params(0)
        e.set_params(p)
        e.reset(2, _abi.MP_SCENE_CUBE_DROP)
        assert b.launch()[1] == torch.cuda.get_device_properties(0).multi_processor_count
        pos = np.ones((5, 4), np.float32)
        for far in (box - 0.1, 0.2):
            pos[:, :3] = [[0.1] * 3, [far] * 3, [0.1] * 3, [far] * 3, [5.0] * 3]
            b.write(_abi.MP_BUF_POSITIONS, pos)
            b.write(_abi.MP_BUF_VELOCITIES, np.zeros_like(pos))
            e.set_positions(pos[:2])
            e.set_velocities(np.zeros_like(pos[:2]))
            for _ in range(3):
                b.step()
                e.step(1.0 / 120.0)
            assert b.check_errors() == 0 and e.check_errors() == 0
            np.testing.assert_array_equal(b.positions()[:2], e.positions())
            np.testing.assert_array_equal(b.velocities()[:2], e.velocities())
    finally:
        b.close()
        e.close()
