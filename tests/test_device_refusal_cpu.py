"""A node on a device that is not a CUDA device is refused before anything is
launched: its tensors' host addresses must not reach a kernel."""

import pytest
import torch

from maddening_b200 import LBMNode, _lib, pipe


class _NoLaunch:
    """The native library without its launching calls."""

    def __init__(self, real):
        self._real = real

    def __getattr__(self, name):
        if not name.endswith("_bytes"):
            raise AssertionError(f"{name} reached with host tensors")
        return getattr(self._real, name)


@pytest.fixture
def cuda_by_name(monkeypatch):
    """CUDA looks available to the nodes made in the test; nothing may launch."""
    def arm():
        real, real_pipe = _NoLaunch(_lib.lib()), _NoLaunch(pipe._lib_pipe())
        monkeypatch.setattr(_lib, "lib", lambda: real)
        monkeypatch.setattr(pipe, "_lib_pipe", lambda: real_pipe)
        monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
        monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
        monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda i: 0, raising=False)
    return arm


@pytest.mark.parametrize("call", ["initial_state", "update", "run", "history", "rollout",
                                  "mass_momentum"])
def test_node_refuses_a_host_device(cuda_by_name, call):
    node = LBMNode("n", 1.0, grid_shape=(4, 5, 6), device="cpu")
    state = {"f": torch.ones(4, 5, 6, 19)}
    cuda_by_name()
    calls = {"initial_state": node.initial_state,
             "update": lambda: node.update(state, {}, 1.0),
             "run": lambda: node.run(state, {}, 2),
             "history": lambda: node.run_with_history(state, {}, 2),
             "rollout": lambda: node.rollout(state, {}, 2),
             "mass_momentum": lambda: node.mass_momentum(state["f"])}
    with pytest.raises(ValueError, match="Expected a cuda device"):
        calls[call]()


def test_pipe_node_refuses_a_host_device(cuda_by_name):
    node = pipe.LBMPipeNode("p", 1.0, nx=12, ny=8, nz=8, device="cpu")
    state = {"f": torch.ones(12, 8, 8, 19), "tracer_f": torch.ones(12, 8, 8, 7),
             "density": torch.ones(12, 8, 8), "tracer": torch.ones(12, 8, 8),
             "velocity": torch.zeros(12, 8, 8, 3)}
    cuda_by_name()
    with pytest.raises(ValueError, match="Expected a cuda device"):
        node.update(state, {}, 1.0)
