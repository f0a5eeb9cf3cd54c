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
