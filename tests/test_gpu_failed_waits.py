"""A wait of the one-pass kernel that runs out must show in the results: the cells
of the block that gave up are NaN in every output, and what later steps and the
tracer compute from them.  The waits run out through the plan's test hook, which
issues no copies, in every block."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda")


def _hooked(shape, storage, steps):
    """Outputs of `steps` steps with a plan whose one-pass waits run out."""
    from maddening_b200 import LBMNode, _lib
    Q = 19 if len(shape) == 3 else 9
    node = LBMNode("t", 1.0, grid_shape=shape, viscosity=0.06, storage=storage,
                   lattice="D3Q19" if Q == 19 else "D2Q9")
    hook = _lib.Plan(Q, shape, node.tau, storage, flags=_lib.PLAN_TEST_WAIT_TIMEOUT)
    st = node.initial_state()
    args, keep = node._step_args(st, {}, DEV)
    f, rho, vel, prs, mom = node._outputs(DEV)
    for x in (f, rho, vel, prs):
        x.fill_(1.0)
    ws = torch.zeros(hook.workspace_bytes(), dtype=torch.uint8, device=DEV)
    _lib.check(_lib.lib().lbm_rollout(
        hook.handle, torch.cuda.current_stream().cuda_stream, st["f"].data_ptr(), f.data_ptr(),
        steps, C.byref(args), C.byref(mom), ws.data_ptr(), ws.numel()))
    torch.cuda.synchronize()
    return f, rho, vel, prs


@pytest.mark.parametrize("shape,storage", [((20, 10, 36), "f32"), ((7, 13, 8), "f16"),
                                           ((20, 37), "f32"), ((9, 256), "bf16")])
def test_update_outputs_are_nan(shape, storage):
    for x in _hooked(shape, storage, 1):
        assert torch.isnan(x).all()


@pytest.mark.parametrize("shape,storage", [((20, 10, 36), "f32"), ((7, 13, 8), "bf16"),
                                           ((9, 256), "f16")])
def test_rollout_outputs_are_nan(shape, storage):
    for x in _hooked(shape, storage, 4):
        assert torch.isnan(x).all()


def test_pipe_update_outputs_are_nan():
    from maddening_b200 import _lib, pipe
    node = pipe.LBMPipeNode("p", 1.0, nx=12, ny=10, nz=32, propeller_x=6)
    st = node.initial_state()
    shape = (12, 10, 32)
    hook = _lib.Plan(19, shape, 0.8, "f32", flags=_lib.PLAN_TEST_WAIT_TIMEOUT)
    wall = torch.as_tensor(node._wall_np.astype("uint8"), device=DEV)
    a = pipe.lbm_pipe_args()
    a.wall, a.propeller, a.tau_tracer = wall.data_ptr(), None, 0.9
    f, g = st["f"].contiguous(), st["tracer_f"].contiguous()
    f_out, g_out, tracer = torch.ones_like(f), torch.ones_like(g), torch.ones(shape, device=DEV)
    rho, vel = torch.ones(shape, device=DEV), torch.ones(shape + (3,), device=DEV)
    m = _lib.lbm_moments()
    m.density, m.velocity = rho.data_ptr(), vel.data_ptr()
    lib = pipe._lib_pipe()
    ws = torch.zeros(hook._size(lib.lbm_pipe_workspace_bytes), dtype=torch.uint8, device=DEV)
    _lib.check(lib.lbm_pipe_rollout(
        hook.handle, torch.cuda.current_stream().cuda_stream, f.data_ptr(), f_out.data_ptr(),
        g.data_ptr(), g_out.data_ptr(), 1, C.byref(a), C.byref(m), tracer.data_ptr(),
        ws.data_ptr(), ws.numel()))
    torch.cuda.synchronize()
    for x in (f_out, rho, vel):
        assert torch.isnan(x).all()
    # a fluid cell whose neighbours are all fluid received only collided populations
    fluid = wall == 0
    inner = fluid.clone()
    for ax in range(3):
        inner &= fluid.roll(1, ax) & fluid.roll(-1, ax)
    assert inner.any() and torch.isnan(tracer[inner]).all() and torch.isnan(g_out[inner]).any(-1).all()
