"""The one-pass step at the edges of its tiles: rows of one cell group less or
more than a tile, row counts around its rows, against the two-pass path (the
same arithmetic, so bit for bit)."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 9, 28), (4, 10, 32), (6, 11, 36), (3, 21, 64),
                                   (5, 248), (4, 252), (6, 256), (3, 380), (7, 504), (5, 508)])
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
