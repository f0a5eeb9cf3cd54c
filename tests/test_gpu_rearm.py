"""A batch whose step was stopped at any of its grid barriers works again once
its error has been read: new positions and velocities (no reset, no restore) step
exactly like a fresh batch's.  What a step expects clean of the one before it
(cell counts, the scenes' bounding boxes) is left dirty by a stopped one."""
import ctypes as C

import numpy as np
import pytest

from mtlphys_b200 import _abi, configs
from mtlphys_b200.batch import Batch

pytestmark = pytest.mark.gpu

SHORT = 2000  # polls: a wait of ~0.1-2 ms


def small_batch():
    w = configs.batch_cubes(num=3, lo=2000, hi=9000)
    b = Batch(0)
    b.reset(w.counts, w.params, w.dts, w.scenes, w.descs)
    return b


def stepped(b, pos, vel, steps=2):
    b.write(_abi.MP_BUF_POSITIONS, pos)
    b.write(_abi.MP_BUF_VELOCITIES, vel)
    for _ in range(steps):
        b.step()
    assert b.check_errors() == 0
    return b.positions(), b.velocities(), b.read(_abi.MP_BUF_SORTED_INDEX)


# barriers of a step: boxes, counts, tile sums, scan, scatter, gather, then the solver's
@pytest.mark.parametrize("passed", [0, 1, 2, 3, 4, 5, 7])
def test_a_stopped_step_leaves_nothing_behind(cuda, passed):
    lib = _abi.load()
    b, ref = small_batch(), small_batch()
    try:
        pos, vel = b.positions(), b.velocities()
        want = stepped(ref, pos, vel)
        far = pos.copy()
        far[:, :3] += np.float32(1.7)  # the stopped step's boxes and counts: other cells
        b.write(_abi.MP_BUF_POSITIONS, far)
        lib.mp_set_spin_limit(SHORT)
        assert lib.mp_batch_debug_barrier_extra(b._h, 1) == _abi.MP_OK
        assert lib.mp_batch_debug_barrier_pass(b._h, passed) == _abi.MP_OK
        b.step()
        bits = C.c_uint32()
        assert lib.mp_batch_check_errors(b._h, C.byref(bits)) == _abi.MP_ERR_SPIN_LIMIT
        lib.mp_set_spin_limit(0)
        assert lib.mp_batch_debug_barrier_extra(b._h, 0) == _abi.MP_OK
        for got, exp in zip(stepped(b, pos, vel), want):
            np.testing.assert_array_equal(got, exp)
    finally:
        lib.mp_set_spin_limit(0)
        b.close()
        ref.close()


@pytest.mark.parametrize("passed", [0, 3, 6, 9])
def test_a_backward_pass_whose_recorded_step_stops_can_be_repeated(cuda, passed):
    """The adjoint kernels that follow a stopped step stay inside their arrays (the
    record is a new one, then one that holds other steps), and the same rollout gives
    its gradients once the error has been read."""
    import torch

    lib = _abi.load()
    b = small_batch()
    try:
        n = b.particle_count()
        g = torch.from_numpy(np.random.default_rng(4).normal(size=(n, 4)).astype(np.float32)).cuda()

        def stop():
            lib.mp_set_spin_limit(SHORT)
            assert lib.mp_batch_debug_barrier_extra(b._h, 1) == _abi.MP_OK
            assert lib.mp_batch_debug_barrier_pass(b._h, passed) == _abi.MP_OK
            b.rollout_backward(g, g)
            assert lib.mp_batch_check_errors(b._h, None) == _abi.MP_ERR_SPIN_LIMIT
            lib.mp_set_spin_limit(0)
            assert lib.mp_batch_debug_barrier_extra(b._h, 0) == _abi.MP_OK

        b.rollout_forward(4, 2)
        end = b.positions()
        stop()
        first = [t.cpu().numpy() for t in b.rollout_backward(g, g)]
        assert b.check_errors() == 0
        stop()
        again = [t.cpu().numpy() for t in b.rollout_backward(g, g)]
        assert b.check_errors() == 0
        for x, y in zip(first, again):
            assert np.isfinite(x).all()
            np.testing.assert_array_equal(x, y)
        np.testing.assert_array_equal(end, b.positions())
    finally:
        lib.mp_set_spin_limit(0)
        b.close()
