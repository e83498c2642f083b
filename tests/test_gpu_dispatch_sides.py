"""Branches of the dispatch that the nodes reach only on large lattices, or not at
all: FP32 pairs with faces by default, and a pipe step without a velocity output."""

import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1024, 1024), (760, 702), (162, 162, 162)])
def test_large_fp32_with_faces_equals_one_cell_per_thread(shape):
    """From 2^19 cells (D2Q9) and 2^22 (D3Q19) FP32 takes pairs."""
    from maddening_b200 import LBMNode
    rng = np.random.default_rng(3)
    kw = dict(grid_shape=shape, viscosity=0.05, outlet_condition="zero_gradient",
              lattice="D3Q19" if len(shape) == 3 else "D2Q9", wall_mask=rng.random(shape) < 0.1)
    a, b = LBMNode("a", 1.0, **kw), LBMNode("b", 1.0, cells_per_thread=1, **kw)
    st = a.initial_state()
    gen = torch.Generator(device="cuda").manual_seed(4)
    st["f"] = st["f"] * (1 + 1e-3 * torch.randn(st["f"].shape, device="cuda", generator=gen))
    bi = {"inlet_velocity": np.array([0.04] + [0.0] * (len(shape) - 1))}
    x, y = a.run(st, bi, 4), b.run(st, bi, 4)
    for key in ("f", "density", "velocity", "pressure"):
        assert torch.equal(x[key], y[key]), key


@pytest.mark.parametrize("shape", [(12, 10, 32), (9, 8, 30)])  # one pass; the pull step
def test_pipe_step_without_a_velocity_output(shape):
    from maddening_b200 import _lib, pipe
    dev = torch.device("cuda")
    node = pipe.LBMPipeNode("p", 1.0, nx=shape[0], ny=shape[1], nz=shape[2], gravity=-2e-5,
                            propeller_x=6, initial_velocity=0.01)
    st = node.initial_state()
    noise = torch.as_tensor(1 + 1e-3 * np.random.default_rng(5).standard_normal(shape + (1,)),
                            device=dev)
    f, g = (st["f"] * noise).float(), (st["tracer_f"] * noise).float()
    wall = torch.as_tensor(node._wall_np.astype("uint8"), device=dev)
    a = pipe.lbm_pipe_args()
    a.wall, a.propeller, a.gravity, a.tau_tracer = wall.data_ptr(), None, -2e-5, 0.9
    lib, outs = pipe._lib_pipe(), []
    for with_velocity in (True, False):
        f_out, g_out = torch.empty_like(f), torch.empty_like(g)
        rho, vel = torch.empty(shape, device=dev), torch.empty(shape + (3,), device=dev)
        tracer = torch.empty(shape, device=dev)
        m = _lib.lbm_moments()
        m.density, m.velocity = rho.data_ptr(), vel.data_ptr() if with_velocity else None
        ws = torch.empty(node._plan._size(lib.lbm_pipe_workspace_bytes), dtype=torch.uint8,
                         device=dev)
        _lib.check(lib.lbm_pipe_rollout(
            node._plan.handle, torch.cuda.current_stream().cuda_stream, f.data_ptr(),
            f_out.data_ptr(), g.data_ptr(), g_out.data_ptr(), 1, C.byref(a), C.byref(m),
            tracer.data_ptr(), ws.data_ptr(), ws.numel()))
        outs.append((f_out, g_out, rho, tracer))
    for x, y in zip(*outs):
        assert torch.equal(x, y)
