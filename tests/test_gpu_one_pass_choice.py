"""Which D2Q9 updates take the one-pass kernel: not the ones on which two passes
are faster, unless the plan asks for it; and the forced one-pass kernel against two
passes on those lattices (the same arithmetic, so bit for bit)."""

import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _takes_one_pass(node):
    """True when one update leaves the workspace untouched but for its status word."""
    from maddening_b200 import _lib
    st, dev = node.initial_state(), torch.device("cuda")
    args, keep = node._step_args(st, {}, dev)
    f, _r, _v, _p, mom = node._outputs(dev)
    ws = torch.full((node.plan.state_bytes(),), 0x55, dtype=torch.uint8, device=dev)
    _lib.check(_lib.lib().lbm_update(
        node.plan.handle, torch.cuda.current_stream().cuda_stream, st["f"].data_ptr(),
        f.data_ptr(), C.byref(args), C.byref(mom), ws.data_ptr(), ws.numel()))
    return bool((ws[4:] == 0x55).all())


@pytest.mark.parametrize("shape,default", [
    ((2000, 3), False), ((300000, 1), False), ((33, 37), False), ((255, 255), False),
    ((1049, 999), False), ((1650, 999), True), ((2100, 2047), True),      # any row length
    ((64, 64), False), ((16384, 256), False), ((1024, 1024), False),
    ((1100, 1000), True), ((2048, 2048), True)])                          # rows of 4 cells
def test_small_or_badly_filled_lattices_take_two_passes(shape, default):
    from maddening_b200 import LBMNode
    for one_pass, want in ((None, default), (True, True), (False, False)):
        node = LBMNode("c", 1.0, grid_shape=shape, viscosity=0.06, lattice="D2Q9",
                       one_pass=one_pass)
        assert _takes_one_pass(node) == want, one_pass


@pytest.mark.parametrize("shape", [(2, 1), (5, 2), (7, 3), (3, 4), (5, 248), (4, 252), (6, 253),
                                   (5, 255), (6, 256), (3, 380), (7, 505), (5, 508)])
@pytest.mark.parametrize("storage", ["f32", "bf16"])
@pytest.mark.parametrize("drive", ["force", "faces"])
def test_forced_one_pass_equals_two_passes(shape, storage, drive):
    from maddening_b200 import LBMNode
    if drive == "faces" and shape[1] < 3:
        pytest.skip("a zero-gradient face needs three cells")
    rng = np.random.default_rng(7)
    kw = dict(grid_shape=shape, viscosity=0.06, lattice="D2Q9", storage=storage,
              wall_mask=rng.random(shape) < 0.15)
    bi = {"body_force": rng.uniform(-1e-5, 1e-5, shape + (2,)).astype(np.float32)}
    if drive == "faces":
        kw.update(inlet_face="y_max", outlet_face="y_min", outlet_condition="zero_gradient")
        bi = {"inlet_velocity": np.array([0.0, -0.03])}
    a, b = LBMNode("a", 1.0, one_pass=True, **kw), LBMNode("b", 1.0, one_pass=False, **kw)
    st = a.initial_state()
    st["f"] = torch.as_tensor(a.lattice.w * (1 + 1e-3 * rng.standard_normal(
        shape + (9,))), device="cuda").to(st["f"].dtype)
    for x, y in ((a.update(st, bi, 1.0), b.update(st, bi, 1.0)),
                 (a.run(st, bi, 3), b.run(st, bi, 3))):
        for key in ("f", "density", "velocity", "pressure"):
            assert torch.equal(x[key], y[key]), key


def test_one_pass_and_two_passes_exclude_each_other():
    from maddening_b200 import _lib
    with pytest.raises(_lib.LbmError, match="one pass and for two"):
        _lib.Plan(9, (8, 8), 0.8, "f32", flags=_lib.PLAN_ONE_PASS | _lib.PLAN_TWO_PASS)
