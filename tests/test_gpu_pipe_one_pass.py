"""A single pipe-node update with its fluid half in one pass against the same
update from populations that are not 16-byte aligned, which takes the pull
step: the same bytes."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 9, 28), (12, 10, 32), (13, 21, 36), (12, 8, 68), (11, 4, 4)])
@pytest.mark.parametrize("gravity", [0.0, -2e-5])
def test_one_pass_pipe_update_equals_the_pull_step(shape, gravity):
    from maddening_b200.pipe import LBMPipeNode
    node = LBMPipeNode("p", 1.0, nx=shape[0], ny=shape[1], nz=shape[2], gravity=gravity,
                       propeller_x=10, propeller_strength=3e-4, initial_velocity=0.01)
    st = node.initial_state()
    rng = np.random.default_rng(4)
    for key in ("f", "tracer_f"):
        noise = torch.as_tensor(1 + 1e-3 * rng.standard_normal(tuple(st[key].shape)), device="cuda")
        st[key] = (st[key] * noise).float().contiguous()
    shifted = torch.empty(st["f"].numel() + 1, device="cuda")[1:].view(st["f"].shape)
    shifted.copy_(st["f"])
    assert shifted.data_ptr() % 16 != 0 and st["f"].data_ptr() % 16 == 0
    a = node.update(st, {}, 1.0)
    b = node.update({**st, "f": shifted}, {}, 1.0)
    for key in ("f", "density", "velocity", "tracer", "tracer_f"):
        assert torch.equal(a[key], b[key]), key
