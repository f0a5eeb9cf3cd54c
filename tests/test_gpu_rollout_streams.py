"""Rollouts on streams that do not wait for the default one."""
import numpy as np
import pytest

from mtlphys_b200 import configs
from mtlphys_b200.batch import Batch

pytestmark = pytest.mark.gpu


def test_the_first_backward_pass_on_a_side_stream(cuda):
    """The rollout's buffers are cleared on the stream that the pass runs on."""
    import torch

    w = configs.diff_cube(side=30)
    grads = []
    for stream in (torch.cuda.default_stream(), torch.cuda.Stream(), torch.cuda.Stream()):
        b = Batch(0)
        try:
            b.reset([w.n], w.params, [w.dt], [w.scene], [w.desc])
            with torch.cuda.stream(stream):
                g = torch.ones((w.n, 4), dtype=torch.float32, device="cuda")
                b.rollout_forward(10, 10, stream)
                out = b.rollout_backward(g, g, stream)
            stream.synchronize()
            grads.append([t.cpu().numpy() for t in out])
            assert b.check_errors() == 0
        finally:
            b.close()
    for other in grads[1:]:
        for x, y in zip(grads[0], other):
            np.testing.assert_array_equal(x, y)
