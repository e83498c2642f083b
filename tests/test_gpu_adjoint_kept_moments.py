"""Gradients from kept moments (short rollouts) against gradients from
checkpoints and recomputed segments: the same reverse kernels on the same
moments, so bit for bit, a second backward pass included."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 7, 9), (8, 4, 36), (13, 11)])
@pytest.mark.parametrize("storage", ["f32", "f64"])
@pytest.mark.parametrize("force_kind", ["field", "uniform", "none"])
def test_kept_moments_give_the_checkpointed_gradients(shape, storage, force_kind):
    from maddening_b200 import LBMNode
    D, steps = len(shape), 30
    rng = np.random.default_rng(2)
    node = LBMNode("g", 1.0, grid_shape=shape, viscosity=0.06, storage=storage,
                   lattice="D3Q19" if D == 3 else "D2Q9", wall_mask=rng.random(shape) < 0.2)
    st = node.initial_state()
    f0 = torch.as_tensor(node.lattice.w * (1 + 1e-3 * rng.standard_normal(
        shape + (node.lattice.Q,))), device="cuda").to(st["f"].dtype)
    force = {"field": rng.uniform(-1e-4, 1e-4, shape + (D,)),
             "uniform": np.array([1e-4, -2e-5, 3e-5][:D]), "none": None}[force_kind]
    weight = torch.as_tensor(rng.standard_normal(f0.shape), device="cuda").to(f0.dtype)

    def gradients(every):
        state = {"f": f0.clone().requires_grad_(True), "wall_mask": st["wall_mask"]}
        wrt, bi = [state["f"]], {}
        if force is not None:
            bi["body_force"] = torch.tensor(force, device="cuda",
                                            dtype=f0.dtype).requires_grad_(True)
            wrt.append(bi["body_force"])
        out = node.rollout(state, bi, steps, checkpoint_every=every)
        loss = (out["velocity"] ** 2).sum() + (weight * out["f"]).sum()
        return [torch.autograd.grad(loss, wrt, retain_graph=True) for _ in range(2)]

    # one segment: kept whole; three segments of 10 steps take less room: recomputed
    kept, segments = gradients(steps), gradients(10)
    for g in (kept[1], segments[0], segments[1]):
        for x, y in zip(kept[0], g):
            assert torch.equal(x, y)
