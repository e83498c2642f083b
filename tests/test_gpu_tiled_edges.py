"""The one-pass step at the edges of its tiles: rows of one cell group (or one
cell) less or more than a tile, row counts around its rows, against the two-pass
path (the same arithmetic, so bit for bit)."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 9, 28), (4, 10, 32), (6, 11, 36), (3, 21, 64),
                                   (5, 248), (4, 252), (6, 256), (3, 380), (7, 504), (5, 508),
                                   # rows that are not groups of four cells: word copies
                                   (5, 251), (4, 253), (3, 3), (6, 505)])
@pytest.mark.parametrize("storage", ["f32", "bf16"])
@pytest.mark.parametrize("drive", ["force", "faces"])
def test_one_pass_at_tile_edges(shape, storage, drive):
    from maddening_b200 import LBMNode
    D = len(shape)
    rng = np.random.default_rng(7)
    kw = dict(grid_shape=shape, viscosity=0.06, lattice="D3Q19" if D == 3 else "D2Q9",
              wall_mask=rng.random(shape) < 0.15, storage=storage)
    bi = {"body_force": rng.uniform(-1e-5, 1e-5, shape + (D,)).astype(np.float32)}
    if drive == "faces":  # on the row axis: the first and the last cell of each row
        last = "z" if D == 3 else "y"
        kw.update(inlet_face=f"{last}_max", outlet_face=f"{last}_min",
                  outlet_condition="zero_gradient")
        bi = {"inlet_velocity": np.array([0.0] * (D - 1) + [-0.03])}
    a, b = LBMNode("a", 1.0, **kw), LBMNode("b", 1.0, one_pass=False, **kw)
    st = a.initial_state()
    st["f"] = torch.as_tensor(a.lattice.w * (1 + 1e-3 * rng.standard_normal(
        shape + (a.lattice.Q,))), device="cuda").to(st["f"].dtype)
    for x, y in ((a.update(st, bi, 1.0), b.update(st, bi, 1.0)), (a.run(st, bi, 2), b.run(st, bi, 2))):
        for key in ("f", "density", "velocity", "pressure"):
            assert torch.equal(x[key], y[key]), key


def test_word_copy_waits_run_out_too():
    """No copy issued: the word-copy form's waits give up, set the status word and
    return; the next call runs normally."""
    import ctypes as C

    from maddening_b200 import LBMNode, _lib
    shape = (20, 37)
    node = LBMNode("t", 1.0, grid_shape=shape, viscosity=0.06, lattice="D2Q9")
    hook = _lib.Plan(9, shape, node.tau, "f32", flags=_lib.PLAN_TEST_WAIT_TIMEOUT)
    st, dev = node.initial_state(), torch.device("cuda")
    args, keep = node._step_args(st, {}, dev)
    f_out, _r, _v, _p, mom = node._outputs(dev)
    ws = torch.full((node.plan.state_bytes(),), 0x55, dtype=torch.uint8, device=dev)
    stream = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.lib().lbm_update(hook.handle, stream, st["f"].data_ptr(), f_out.data_ptr(),
                                     C.byref(args), C.byref(mom), ws.data_ptr(), ws.numel()))
    torch.cuda.synchronize()
    assert int(ws[:4].view(torch.int32).item()) == 1
    two = LBMNode("t", 1.0, grid_shape=shape, viscosity=0.06, lattice="D2Q9", one_pass=False)
    assert torch.equal(node.update(st, {}, 1.0)["f"], two.update(st, {}, 1.0)["f"])
