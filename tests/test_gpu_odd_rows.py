"""Rollouts with 16-bit state and odd rows: padded state rows and two cells per
thread give the one-cell form's bytes, and so does a call whose workspace has
no room for the padding."""

import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 3, 1), (5, 4, 3), (3, 5, 63), (6, 7, 129), (9, 1), (8, 257)])
@pytest.mark.parametrize("storage", ["f16", "bf16"])
@pytest.mark.parametrize("drive", ["none", "field", "faces"])
def test_odd_rows_equal_the_one_cell_form(shape, storage, drive):
    from maddening_b200 import LBMNode, _lib
    D = len(shape)
    rng = np.random.default_rng(11)
    kw = dict(grid_shape=shape, viscosity=0.05, lattice="D3Q19" if D == 3 else "D2Q9",
              wall_mask=rng.random(shape) < 0.15, storage=storage)
    bi = {}
    if drive == "field":
        bi = {"body_force": rng.uniform(-1e-5, 1e-5, shape + (D,)).astype(np.float32)}
    elif drive == "faces":
        kw.update(outlet_condition="zero_gradient")
        bi = {"inlet_velocity": np.array([0.04] + [0.0] * (D - 1))}
    two, one = LBMNode("a", 1.0, **kw), LBMNode("b", 1.0, cells_per_thread=1, **kw)
    st = two.initial_state()
    st["f"] = torch.as_tensor(two.lattice.w * (1 + 1e-3 * rng.standard_normal(
        shape + (two.lattice.Q,))), device="cuda").to(st["f"].dtype)
    x, y = two.run(st, bi, 6), one.run(st, bi, 6)
    for key in ("f", "density", "velocity", "pressure"):
        assert torch.equal(x[key], y[key]), key
    # two unpadded state copies and the status word: the room this call needs at least
    dev = torch.device("cuda")
    args, keep = two._step_args(st, bi, dev)
    f, rho, _v, _p, mom = two._outputs(dev)
    need = 2 * ((two.plan.state_bytes() + 255) // 256 * 256) + 256
    ws = torch.empty(need, dtype=torch.uint8, device=dev)
    _lib.check(_lib.lib().lbm_rollout(
        two.plan.handle, torch.cuda.current_stream().cuda_stream, st["f"].data_ptr(),
        f.data_ptr(), 6, C.byref(args), C.byref(mom), ws.data_ptr(), ws.numel()))
    assert torch.equal(f, y["f"]) and torch.equal(rho, y["density"])
