"""Which rollouts with 16-bit state and odd rows keep padded rows and two cells per
thread: not small lattices with faces or lattices of very short rows, on which one
cell per thread is faster; and the forced pairs against one cell per thread."""

import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _node(shape, storage, faces, cells, wall=None):
    from maddening_b200 import LBMNode
    kw = dict(outlet_condition="zero_gradient") if faces else {}
    bi = {"inlet_velocity": np.array([0.03] + [0.0] * (len(shape) - 1))} if faces else {}
    return LBMNode("c", 1.0, grid_shape=shape, viscosity=0.05, storage=storage, wall_mask=wall,
                   lattice="D3Q19" if len(shape) == 3 else "D2Q9", cells_per_thread=cells,
                   **kw), bi


def _keeps_padded_rows(node, bi):
    """True when a rollout with room for padded rows writes behind two unpadded copies."""
    from maddening_b200 import _lib
    st, dev = node.initial_state(), torch.device("cuda")
    args, keep = node._step_args(st, bi, dev)
    f, _r, _v, _p, mom = node._outputs(dev)
    plain = 2 * ((node.plan.state_bytes() + 255) // 256 * 256) + 256
    ws = torch.full((node.plan.workspace_bytes() + 4096,), 0x55, dtype=torch.uint8, device=dev)
    _lib.check(_lib.lib().lbm_rollout(
        node.plan.handle, torch.cuda.current_stream().cuda_stream, st["f"].data_ptr(),
        f.data_ptr(), 3, C.byref(args), C.byref(mom), ws.data_ptr(), ws.numel()))
    return bool((ws[plain:] != 0x55).any())


@pytest.mark.parametrize("shape,faces,default", [
    ((33, 33, 33), True, False), ((64, 64, 63), True, False), ((80, 80, 81), True, True),
    ((200, 200, 15), True, False), ((300, 301), True, False), ((700, 701), True, True),
    ((33, 33, 33), False, True), ((24, 24, 25), False, False), ((256, 256, 1), False, False),
    ((200, 200, 5), False, True), ((600, 600, 5), False, False), ((100000, 1), False, False)])
def test_where_rows_are_padded(shape, faces, default):
    for cells, want in ((None, default), (1, False), (2, True)):
        assert _keeps_padded_rows(*_node(shape, "f16", faces, cells)) == want, cells


@pytest.mark.parametrize("shape", [(4, 3, 1), (5, 4, 3), (3, 5, 63), (6, 7, 129), (9, 1), (8, 257)])
@pytest.mark.parametrize("storage", ["f16", "bf16"])
@pytest.mark.parametrize("drive", ["none", "field", "faces"])
def test_forced_pairs_equal_the_one_cell_form(shape, storage, drive):
    rng = np.random.default_rng(11)
    wall = rng.random(shape) < 0.15
    two, bi = _node(shape, storage, drive == "faces", 2, wall)
    one, _ = _node(shape, storage, drive == "faces", 1, wall)
    if drive == "field":
        bi = {"body_force": rng.uniform(-1e-5, 1e-5, shape + (len(shape),)).astype(np.float32)}
    st = two.initial_state()
    st["f"] = torch.as_tensor(two.lattice.w * (1 + 1e-3 * rng.standard_normal(
        shape + (two.lattice.Q,))), device="cuda").to(st["f"].dtype)
    x, y = two.run(st, bi, 6), one.run(st, bi, 6)
    for key in ("f", "density", "velocity", "pressure"):
        assert torch.equal(x[key], y[key]), key
