"""Rollouts with 16-bit state in a workspace off 4-byte boundaries: no paired
access may be taken there, and the outputs are those of an aligned workspace."""

import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 4, 3), (6, 7, 129), (4, 6, 66), (9, 1), (8, 257), (6, 130)])
@pytest.mark.parametrize("storage", ["f16", "bf16"])
@pytest.mark.parametrize("cells", [None, 2])
def test_workspace_on_a_two_byte_boundary(shape, storage, cells):
    from maddening_b200 import LBMNode, _lib
    rng = np.random.default_rng(5)
    node = LBMNode("w", 1.0, grid_shape=shape, viscosity=0.05, storage=storage,
                   cells_per_thread=cells,
                   lattice="D3Q19" if len(shape) == 3 else "D2Q9",
                   wall_mask=rng.random(shape) < 0.15)
    st, dev = node.initial_state(), torch.device("cuda")
    st["f"] = torch.as_tensor(node.lattice.w * (1 + 1e-3 * rng.standard_normal(
        shape + (node.lattice.Q,))), device=dev).to(st["f"].dtype)
    ref = node.run(st, {}, 6)
    args, keep = node._step_args(st, {}, dev)
    f, rho, _v, _p, mom = node._outputs(dev)
    ws = torch.empty(node.plan.workspace_bytes() + 2, dtype=torch.uint8, device=dev)[2:]
    assert ws.data_ptr() % 4 == 2
    _lib.check(_lib.lib().lbm_rollout(
        node.plan.handle, torch.cuda.current_stream().cuda_stream, st["f"].data_ptr(),
        f.data_ptr(), 6, C.byref(args), C.byref(mom), ws.data_ptr(), ws.numel()))
    assert torch.equal(f, ref["f"]) and torch.equal(rho, ref["density"])
