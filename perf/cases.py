"""The work a program has this framework do, as a set of measurable cases.

Each case is one call (or a forward and a backward call) of a public entry
point with inputs of its own: single node steps as a graph manager drives
them, fused rollouts in every storage type, a differentiated rollout, a batched
ensemble and the pipe node in both of its modes.  ``listed`` are fixed sizes,
``draw`` gives other sizes, lattices, storages and boundary conditions of the
same ranges.  ``exact`` is the same physics in plain torch float64.
"""

import math

import numpy as np
import torch

from maddening_b200 import LBMNode
from maddening_b200.batched import LBMEnsemble
from maddening_b200.pipe import LBMPipeNode

_E3 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1),
       (1, 1, 0), (-1, 1, 0), (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1),
       (-1, 0, -1), (0, 1, 1), (0, -1, 1), (0, 1, -1), (0, -1, -1)]
_E2 = [(0, 0), (1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (-1, 1), (1, -1), (-1, -1)]
_W3 = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
_W2 = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4
_W7 = [1 / 4] + [1 / 8] * 6


def _sets(D):
    e, w = (_E3, _W3) if D == 3 else (_E2, _W2)
    opp = [e.index(tuple(-c for c in v)) for v in e]
    return e, w, opp


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # One step of the node at its default grid, driven by pressures: what a
        # graph manager calls once per time step of a small coupled model.
        {"name": "step_default_grid", "kind": "step", "shape": "64x32x32", "storage": "f32",
         "walls": "channel", "drive": "pressure"},
        # One step in a vessel-like mask with odd extents (a voxelised geometry
        # gives whatever extents its bounding box has).
        {"name": "step_vessel_odd_grid", "kind": "step", "shape": "151x75x70", "storage": "f32",
         "walls": "vessel", "drive": "pressure"},
        # One step of a large obstacle flow, velocity inlet and open outlet.
        {"name": "step_obstacles_256", "kind": "step", "shape": "256x256x256",
         "storage": "f32", "walls": "spheres", "drive": "inlet"},
        # One step of a large two-dimensional channel under a body force.
        {"name": "step_plane_2048", "kind": "step", "shape": "2048x2048", "storage": "f32",
         "walls": "channel", "drive": "force"},
        # A rollout of the 64^3 channel (a parameter study's usual size).
        {"name": "run_channel_64", "kind": "run", "shape": "64x64x64", "storage": "f32",
         "walls": "channel", "drive": "force", "steps": 100},
        # Rollouts of the large obstacle flow, FP32 state and FP16 state.
        {"name": "run_obstacles_256_f32", "kind": "run", "shape": "256x256x256",
         "storage": "f32", "walls": "spheres", "drive": "inlet", "steps": 20},
        {"name": "run_obstacles_256_f16", "kind": "run", "shape": "256x256x256",
         "storage": "f16", "walls": "spheres", "drive": "inlet", "steps": 20},
        # A rollout under a force field (a coupled magnetic or drag force) on a
        # lattice with odd extents, BF16 state.
        {"name": "run_force_field_bf16", "kind": "run", "shape": "149x111x93",
         "storage": "bf16", "walls": "vessel", "drive": "field", "steps": 20},
        # Forward and backward through a rollout: the gradient of a velocity
        # misfit with respect to the initial state and to a force field.
        {"name": "gradient_96", "kind": "gradient", "shape": "96x96x96", "storage": "f32",
         "walls": "spheres", "drive": "field", "steps": 40},
        # A sweep over uneven lattices advanced together, FP16 state.
        {"name": "ensemble_16_f16", "kind": "ensemble", "members": 16, "lo": 32, "hi": 160,
         "storage": "f16", "steps": 20},
        # One step of the pipe node (fluid and tracer).
        {"name": "pipe_step", "kind": "pipe", "shape": "256x128x128", "storage": "f32",
         "phases": 1, "steps": 1},
        # A two-phase rollout of the pipe node.
        {"name": "pipe_two_phase_run", "kind": "pipe", "shape": "256x128x128",
         "storage": "f32", "phases": 2, "steps": 20},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _extents(rng, D, cells_lo, cells_hi):
    """Extents whose product is log-uniform in [cells_lo, cells_hi], sides within
    a factor of about two of each other, odd ones as likely as even ones; every
    third draw has a last extent that is a multiple of 32."""
    cells = math.exp(rng.uniform(math.log(cells_lo), math.log(cells_hi)))
    side = cells ** (1.0 / D)
    n = [max(16, int(round(side * math.exp(rng.uniform(-0.35, 0.35))))) for _ in range(D)]
    if rng.random() < 1 / 3:
        n[-1] = max(32, 32 * int(round(n[-1] / 32)))
    return "x".join(str(v) for v in n)


def draw(rng):
    kind = rng.choice(["step", "step", "run", "run", "run", "gradient", "ensemble", "pipe"])
    if kind in ("step", "run"):
        D = 3 if rng.random() < 0.7 else 2
        # up to half of the largest listed lattice in 64-bit state
        storage = rng.choice(["f32", "f32", "f16", "bf16", "f64"])
        top = (1.6e7 if D == 3 else 1.2e7) / (2 if storage == "f64" else 1)
        c = {"kind": kind, "shape": _extents(rng, D, 6e4, top), "storage": storage,
             "walls": rng.choice(["channel", "vessel", "spheres"]),
             "drive": rng.choice(["pressure", "inlet", "force", "field"])}
        if kind == "run":
            c["steps"] = rng.randint(2, 20)
        return c
    if kind == "gradient":
        return {"kind": kind, "shape": _extents(rng, rng.choice([2, 3]), 6e4, 9e5),
                "storage": "f32", "walls": rng.choice(["channel", "spheres"]),
                "drive": rng.choice(["force", "field"]), "steps": rng.randint(10, 40)}
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(3, 16), "lo": 32,
                "hi": _log_int(rng, 48, 160), "storage": rng.choice(["f32", "f16", "bf16"]),
                "steps": rng.randint(4, 20)}
    return {"kind": "pipe", "shape": _extents(rng, 3, 6e4, 4e6), "storage": "f32",
            "phases": rng.choice([1, 2]), "steps": rng.choice([1, rng.randint(2, 20)])}


# ---------------------------------------------------------------------------
# Inputs (shared by prepare and exact; nothing of the framework is used)
# ---------------------------------------------------------------------------


def _shape(case):
    return tuple(int(v) for v in case["shape"].split("x"))


def _modes(shape, gen, amp, dev, count=3):
    """A smooth periodic float32 field: a few low Fourier modes with random phases."""
    D = len(shape)
    out = torch.zeros(shape, dtype=torch.float32, device=dev)
    r = torch.rand((count, D + 2), generator=gen).tolist()
    for m in r:
        arg = torch.zeros((1,) * D, device=dev)
        for d in range(D):
            x = torch.arange(shape[d], dtype=torch.float32, device=dev) / shape[d]
            x = (2 * math.pi * int(1 + 3 * m[d])) * x
            arg = arg + x.reshape([-1 if k == d else 1 for k in range(D)])
        out += (amp * (0.3 + m[D])) * torch.sin(arg + 2 * math.pi * m[D + 1])
    return out


def _walls(shape, kind, seed):
    """Wall mask as a host array (True = wall): the two last-axis planes, a
    meandering vessel along axis 0, or a tenth of the cells in random balls."""
    D = len(shape)
    wall = np.zeros(shape, dtype=bool)
    rng = np.random.RandomState(seed % (1 << 31))
    if kind == "channel":
        wall[..., 0] = True
        wall[..., -1] = True
    elif kind == "vessel":
        x = np.arange(shape[0], dtype=np.float64)
        phase = rng.uniform(0, 2 * np.pi, D)
        r2 = 0.0
        for d in range(1, D):
            mid = (shape[d] - 1) / 2.0 + 0.06 * shape[d] * np.sin(
                2 * np.pi * x / shape[0] + phase[d])
            y = np.arange(shape[d], dtype=np.float64)
            t = (y[None, :] - mid[:, None]) / (0.42 * shape[d])
            s = [shape[0]] + [1] * (D - 1)
            s[d] = shape[d]
            r2 = r2 + (t * t).reshape(s)
        wall |= np.broadcast_to(r2 >= 1.0, shape)
    else:
        lo, hi = (4.0, 12.0) if min(shape) >= 64 else (2.0, 5.0)
        solid, total = 0, wall.size
        for _ in range(20000):
            if solid >= 0.1 * total:
                break
            r = rng.uniform(lo, hi)
            c = [rng.uniform(r + 2, max(r + 3, shape[0] - r - 3))]
            c += [rng.uniform(r, max(r + 1, n - r - 1)) for n in shape[1:]]
            box = tuple(slice(max(0, int(a - r)), min(n, int(a + r) + 2))
                        for a, n in zip(c, shape))
            grid = np.ogrid[box]
            ball = sum((g - a) ** 2 for g, a in zip(grid, c)) < r * r
            view = wall[box]
            solid += int(np.count_nonzero(ball & ~view))
            view |= ball
        if D >= 2:
            wall[0] = False
            wall[-1] = False
    return wall


def _feq32(rho, u, gen_seed, dev):
    """float32 populations near equilibrium, in the node's (*grid, Q) layout."""
    D = len(u)
    e, w, _ = _sets(D)
    f = torch.empty(tuple(rho.shape) + (len(e),), dtype=torch.float32, device=dev)
    usq = sum(v * v for v in u)
    g = torch.Generator(device=dev).manual_seed(gen_seed)
    for q, v in enumerate(e):
        eu = sum(float(c) * u[d] for d, c in enumerate(v) if c) if any(v) else 0.0 * usq
        noise = torch.randn(rho.shape, generator=g, device=dev)
        f[..., q] = w[q] * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * usq + 2e-5 * noise)
    return f


def _flow(case, seed, shape, walls, drive):
    """One lattice's inputs: f, wall mask, boundary inputs, tau."""
    dev = _device()
    D = len(shape)
    gen = torch.Generator().manual_seed(seed)
    wall = _walls(shape, walls, seed)
    w = torch.as_tensor(wall, device=dev)
    rho = 1 + _modes(shape, gen, 1e-3, dev)
    u = [torch.where(w, 0.0, _modes(shape, gen, 0.01, dev)) for _ in range(D)]
    if drive in ("inlet", "pressure"):
        u[0] = torch.where(w, 0.0, u[0] + 0.03)
    f = _feq32(rho, u, seed + 1, dev)
    r = torch.rand(8, generator=gen).tolist()
    bi, extra = {}, {}
    if drive == "pressure":
        bi = {"inlet_pressure": (1.0 + 0.004 * r[0]) / 3.0,
              "outlet_pressure": (1.0 - 0.004 * r[1]) / 3.0}
    elif drive == "inlet":
        bi = {"inlet_velocity": np.array([0.03 + 0.03 * r[0]] + [0.0] * (D - 1))}
        extra = {"outlet_condition": "zero_gradient"}
    elif drive == "force":
        bi = {"body_force": np.array([1e-6 + 1e-5 * r[0]] + [1e-7 * v for v in r[1:D]],
                                     dtype=np.float32)}
    else:
        field = torch.stack([_modes(shape, gen, 1e-5, dev) for _ in range(D)], dim=-1)
        bi = {"body_force": field.contiguous()}
    return f, wall, bi, extra, 0.55 + 0.4 * r[6]


def _members(case):
    """Extents, relaxation times and forces of an ensemble's members."""
    rng = np.random.RandomState(1000 + case["members"])
    got = []
    for _ in range(case["members"]):
        shape = tuple(int(round(math.exp(rng.uniform(math.log(case["lo"]),
                                                     math.log(case["hi"]))))) for _ in range(3))
        got.append((shape, float(rng.uniform(0.55, 1.5)), float(rng.uniform(1e-7, 1e-5))))
    return got


_PIPE = {"tau": 0.8, "pipe_radius": 0.9, "propeller_x": 10, "propeller_radius": 0.8,
         "tau_tracer": 0.6}
_MP = {"G": -4.5, "rho_liquid": 1.0, "rho_gas": 0.25, "rho_0": 1.0, "gravity": -1e-5}


def _pipe_masks(shape):
    """Wall and propeller cross sections (float32 radii, as the node defines them)."""
    _, ny, nz = shape
    yy, zz = np.meshgrid(np.arange(ny, dtype=np.float32), np.arange(nz, dtype=np.float32),
                         indexing="ij")
    r = np.sqrt((yy - np.float32((ny - 1) / 2.0)) ** 2 + (zz - np.float32((nz - 1) / 2.0)) ** 2)
    edge = _PIPE["pipe_radius"] * min(ny, nz) / 2.0
    return r >= np.float32(edge), r < np.float32(_PIPE["propeller_radius"] * edge)


def _pipe_inputs(case, seed):
    dev = _device()
    shape = _shape(case)
    gen = torch.Generator().manual_seed(seed)
    wall2, _ = _pipe_masks(shape)
    w = torch.as_tensor(wall2, device=dev)[None].expand(shape)
    u = [torch.where(w, 0.0, _modes(shape, gen, 0.004, dev)) for _ in range(3)]
    if case["phases"] == 2:
        z = torch.arange(shape[2], dtype=torch.float32, device=dev)
        phase = 0.5 * (1 + torch.tanh((0.5 * shape[2] - z) / 5.0))
        rho = _MP["rho_gas"] + (_MP["rho_liquid"] - _MP["rho_gas"]) * phase
        rho = rho.expand(shape) * (1 + _modes(shape, gen, 0.01, dev))
        rho = torch.where(w, _MP["rho_gas"], rho)
        tracer = ((rho - _MP["rho_gas"]) / (_MP["rho_liquid"] - _MP["rho_gas"])).clamp(0, 1)
    else:
        rho = 1 + _modes(shape, gen, 1e-3, dev)
        tracer = (0.5 + _modes(shape, gen, 0.1, dev)).clamp(0, 1)
    tracer = torch.where(w, 0.0, tracer)
    f = _feq32(rho, u, seed + 1, dev)
    g = torch.empty(shape + (7,), dtype=torch.float32, device=dev)
    for q in range(7):
        eu = sum(float(c) * u[d] for d, c in enumerate(_E3[q]) if c) if q else 0.0
        g[..., q] = _W7[q] * tracer * (1 + 3 * eu)
    strength = 5e-4 * (0.5 + float(torch.rand(1, generator=gen)))
    return f, rho, torch.stack(u, dim=-1), tracer, g, strength


def _as_state(f, wall, io):
    f = f.to(io)
    D = f.dim() - 1
    e, _, _ = _sets(D)
    rho = f.sum(-1)
    vel = (f @ torch.tensor(e, dtype=io, device=f.device)) / rho[..., None]
    return {"f": f, "density": rho, "velocity": vel, "pressure": rho / 3.0,
            "wall_mask": torch.as_tensor(wall.astype(np.uint8), device=f.device)}


# ---------------------------------------------------------------------------
# prepare / run / work
# ---------------------------------------------------------------------------


def _node(shape, tau, wall, storage, extra):
    return LBMNode("lbm", 1.0, grid_shape=shape, viscosity=(tau - 0.5) / 3.0,
                   lattice="D3Q19" if len(shape) == 3 else "D2Q9", wall_mask=wall,
                   storage=storage, **extra)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        nodes, states, bis = [], [], []
        for i, (shape, tau, g) in enumerate(_members(case)):
            f, wall, _, _, _ = _flow(case, seed + 17 * i, shape, "channel", "force")
            nodes.append(_node(shape, tau, wall, case["storage"], {}))
            states.append({"f": f})  # the walls are the nodes' own
            bis.append({"body_force": np.array([g, 0, 0], dtype=np.float32)})
        return {"kind": kind, "ens": LBMEnsemble(nodes), "states": states, "bis": bis,
                "steps": case["steps"]}
    if kind == "pipe":
        shape = _shape(case)
        f, rho, vel, tracer, g, strength = _pipe_inputs(case, seed)
        node = LBMPipeNode("pipe", 1.0, nx=shape[0], ny=shape[1], nz=shape[2], **_PIPE,
                           **(_MP if case["phases"] == 2 else {}))
        return {"kind": kind, "node": node, "steps": case["steps"],
                "state": {"f": f, "density": rho, "velocity": vel, "tracer": tracer,
                          "tracer_f": g},
                "bi": {"propeller_force": strength}}
    shape = _shape(case)
    f, wall, bi, extra, tau = _flow(case, seed, shape, case["walls"], case["drive"])
    node = _node(shape, tau, wall, case["storage"], extra)
    state = _as_state(f, wall, torch.float64 if case["storage"] == "f64" else torch.float32)
    s = {"kind": kind, "node": node, "state": state, "bi": bi, "steps": case.get("steps", 1)}
    if kind == "gradient":
        s["target"] = torch.zeros_like(state["velocity"])
        s["f0"] = state["f"].requires_grad_(True)
        force = bi["body_force"]
        if not isinstance(force, torch.Tensor):
            force = torch.as_tensor(force, device=state["f"].device)
        s["force"] = force.requires_grad_(True)
        state["f"] = s["f0"]
    return s


def run(state):
    kind = state["kind"]
    if kind == "ensemble":
        return state["ens"].run(state["states"], state["bis"], state["steps"])
    node = state["node"]
    if kind == "gradient":
        out = node.rollout(state["state"], {"body_force": state["force"]}, state["steps"])
        loss = ((out["velocity"] - state["target"]) ** 2).sum()
        gf, gF = torch.autograd.grad(loss, [state["f0"], state["force"]])
        return {"loss": loss.detach(), "f": out["f"].detach(),
                "velocity": out["velocity"].detach(), "grad_f": gf, "grad_force": gF}
    if kind == "step" or (kind == "pipe" and state["steps"] == 1):
        return node.update(state["state"], state["bi"], 1.0)
    return node.run(state["state"], state["bi"], state["steps"])


def work(case):
    """Bytes and operations of one pass.  A rollout of n steps is n dependent
    sweeps: every step reads and writes each population once, in the type the
    case stores them; inputs (wall mask, force field) and outputs (moments) of
    the call count once."""
    kind, steps = case["kind"], case.get("steps", 1)
    if kind == "ensemble":
        cells = sum(a * b * c for (a, b, c), _, _ in _members(case))
        D = 3
    else:
        cells = math.prod(_shape(case))
        D = len(_shape(case))
    Q = 19 if D == 3 else 9
    pop = {"f32": 4, "f16": 2, "bf16": 2, "f64": 8}[case["storage"]]
    io = 8 if case["storage"] == "f64" else 4
    flops = (250 if Q == 19 else 110) * cells * steps
    if kind == "pipe":
        if case["phases"] == 2:
            # two sweeps per step: the force needs every density first; the
            # tracer populations pass through
            b = steps * (3 * Q * 4 + 2 * 4) + 2 * 7 * 4
            return {"bytes": cells * (b + 20 + 1), "flops": 2 * flops}
        return {"bytes": cells * (steps * 2 * (Q + 7) * 4 + 20 + 1), "flops": flops * 1.2}
    outputs = io * (D + 2) + 1
    if case.get("drive") == "field":
        outputs += io * D
    if kind == "gradient":
        # forward sweep; backward sweep over the adjoint populations with the
        # density and velocity of every step, and the force gradient
        b = steps * (2 * Q * 4 + 2 * Q * 4 + 2 * (D + 1) * 4) + 2 * Q * 4 + 8 * D
        return {"bytes": cells * (b + outputs), "flops": 3 * flops}
    if kind == "step":
        return {"bytes": cells * (2 * Q * io + outputs), "flops": flops}
    return {"bytes": cells * (steps * 2 * Q * pop + outputs), "flops": flops}


# ---------------------------------------------------------------------------
# exact: the same physics in float64
# ---------------------------------------------------------------------------


def _roll(x, e, sign=1):
    for d, c in enumerate(e):
        if c:
            x = torch.roll(x, sign * c, d)
    return x


def _moments64(f, e, F, half=True):
    D = len(e[0])
    rho = sum(f)
    u = []
    for d in range(D):
        m = sum((fq if v[d] > 0 else -fq) for fq, v in zip(f, e) if v[d])
        if F is not None and half:
            m = m + 0.5 * F[d]
        u.append(m / rho.clamp(min=1e-10))
    return rho, u


def _collide64(f, e, w, rho, u, F, tau):
    D = len(e[0])
    usq = sum(v * v for v in u)
    uF = sum(u[d] * F[d] for d in range(D)) if F is not None else None
    out = []
    for q, v in enumerate(e):
        axes = [d for d in range(D) if v[d]]
        eu = sum(v[d] * u[d] for d in axes) if axes else torch.zeros_like(usq)
        r = f[q] - (f[q] - w[q] * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * usq)) / tau
        if F is not None:
            eF = sum(v[d] * F[d] for d in axes) if axes else 0.0
            r = r + (1 - 0.5 / tau) * w[q] * (3 * (eF - uF) + 9 * eu * eF)
        out.append(r)
    return out


def _stream_walls64(p, e, opp, wall):
    s = [_roll(x, v) for x, v in zip(p, e)]
    return [torch.where(wall, s[opp[q]], s[q]) for q in range(len(e))]


def _feq_face(w, v, rho, un, vec=None):
    if vec is None:
        eu, usq = v[0] * un, un * un
    else:
        eu, usq = sum(a * b for a, b in zip(v, vec)), sum(b * b for b in vec)
    return w * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * usq)


def _faces64(f, e, w, opp, wall, bi, zero_gradient):
    """Inlet at the first plane of axis 0, outlet at the last."""
    def pressure(f, at, side, p):
        rho_p = float(p) / (1.0 / 3.0)
        known = sum(f[q][at] for q, v in enumerate(e) if v[0] == 0 or (v[0] > 0) != (side > 0))
        un = side * (1 - known / rho_p)
        for q, v in enumerate(e):
            if v[0] == side:
                o = opp[q]
                new = (f[o][at] + _feq_face(w[q], v, rho_p, un)
                       - _feq_face(w[o], e[o], rho_p, un))
                f[q][at] = torch.where(wall[at], f[q][at], new)

    inner = [fq[-2].clone() for fq in f] if zero_gradient else None
    if "inlet_pressure" in bi:
        pressure(f, 0, 1, bi["inlet_pressure"])
    if "inlet_velocity" in bi:
        vec = [float(x) for x in bi["inlet_velocity"]]
        tang = sum(f[q][0] for q, v in enumerate(e) if v[0] == 0)
        known = sum(f[q][0] for q, v in enumerate(e) if v[0] < 0)
        rho = (tang + 2 * known) / (1 - vec[0])
        for q, v in enumerate(e):
            if v[0] > 0:
                o = opp[q]
                new = (f[o][0] + _feq_face(w[q], v, rho, None, vec)
                       - _feq_face(w[o], e[o], rho, None, vec))
                f[q][0] = torch.where(wall[0], f[q][0], new)
    if zero_gradient:
        for q, v in enumerate(e):
            if v[0] < 0:
                f[q][-1] = torch.where(wall[-1], f[q][-1], inner[q])
    elif "outlet_pressure" in bi:
        pressure(f, -1, -1, bi["outlet_pressure"])
    return f


def _run64(f32, wall, bi, zero_gradient, tau, steps):
    D = f32.dim() - 1
    e, w, opp = _sets(D)
    wm = torch.as_tensor(wall, device=f32.device)
    f = [f32[..., q].double().contiguous() for q in range(len(e))]
    F = bi.get("body_force")
    if isinstance(F, torch.Tensor):
        F = [F[..., d].double() for d in range(D)]
    elif F is not None:
        F = [float(v) for v in F]
    for _ in range(steps):
        rho, u = _moments64(f, e, F)
        f = _stream_walls64(_collide64(f, e, w, rho, u, F, tau), e, opp, wm)
        f = _faces64(f, e, w, opp, wm, bi, zero_gradient)
    rho, u = _moments64(f, e, F)
    vel = torch.stack([torch.where(wm, 0.0, v) for v in u], dim=-1)
    return {"f": torch.stack(f, dim=-1), "density": rho, "velocity": vel, "pressure": rho / 3.0}


def _gradient64(f32, wall, force, tau, steps):
    D = f32.dim() - 1
    e, w, opp = _sets(D)
    wm = torch.as_tensor(wall, device=f32.device)
    F64 = force.detach().double()

    def step(f, F):
        rho, u = _moments64(f, e, F)
        return _stream_walls64(_collide64(f, e, w, rho, u, F, tau), e, opp, wm)

    def parts(F):
        return [F[..., d] for d in range(D)]

    f = [f32.detach()[..., q].double().contiguous() for q in range(len(e))]
    seen = []
    for _ in range(steps):
        seen.append(f)
        f = step(f, parts(F64))
    leaf = [x.requires_grad_(True) for x in f]
    Fl = F64.clone().requires_grad_(True)
    _, u = _moments64(leaf, e, parts(Fl))
    vel = torch.stack([torch.where(wm, 0.0, v) for v in u], dim=-1)
    loss = (vel ** 2).sum()
    *lam, gF = torch.autograd.grad(loss, leaf + [Fl])
    for f in reversed(seen):
        leaf = [x.detach().requires_grad_(True) for x in f]
        Fl = F64.clone().requires_grad_(True)
        *lam, g = torch.autograd.grad(step(leaf, parts(Fl)), leaf + [Fl], lam)
        gF = gF + g
    last = [x.detach() for x in seen[-1]]
    out = step(last, parts(F64))
    return {"loss": loss.detach(), "f": torch.stack(out, dim=-1), "velocity": vel.detach(),
            "grad_f": torch.stack(lam, dim=-1), "grad_force": gF}


def _pipe64(case, seed):
    shape = _shape(case)
    f32, _, _, _, g32, strength = _pipe_inputs(case, seed)
    e, w, opp = _sets(3)
    dev = f32.device
    wall2, prop2 = _pipe_masks(shape)
    wm = torch.as_tensor(wall2, device=dev)[None].expand(shape).contiguous()
    fx = torch.zeros(shape, dtype=torch.float64, device=dev)
    fx[_PIPE["propeller_x"]] = torch.as_tensor(prop2, device=dev).double() * strength
    two = case["phases"] == 2
    fz = torch.where(wm, 0.0, _MP["gravity"] if two else 0.0).double()
    F0 = [fx, torch.zeros_like(fx), fz]
    tau = _PIPE["tau"]
    f = [f32[..., q].double().contiguous() for q in range(19)]
    g = [g32[..., q].double().contiguous() for q in range(7)]
    psi_w = _MP["rho_0"] * (1 - math.exp(-_MP["rho_liquid"] / _MP["rho_0"]))
    for _ in range(case["steps"]):
        rho, u = _moments64(f, e, None)
        if two:
            psi = torch.where(wm, psi_w, -_MP["rho_0"] * torch.expm1(-rho / _MP["rho_0"]))
            F = list(F0)
            for d in range(3):
                grad = sum(v[d] * w[q] * _roll(psi, v, -1) for q, v in enumerate(e) if v[d])
                F[d] = F[d] + torch.where(wm, 0.0, -_MP["G"] * psi * grad)
            us = [u[d] + F[d] / rho.clamp(min=0.01) for d in range(3)]
            mag = torch.sqrt(sum(v * v for v in us))
            us = [v * (0.25 / mag.clamp(min=1e-10)).clamp(max=1.0) for v in us]
            usq, ssq = sum(v * v for v in u), sum(v * v for v in us)
            p = []
            for q, v in enumerate(e):
                def feq(uu, sq, v=v, q=q):
                    eu = sum(v[d] * uu[d] for d in range(3))
                    return w[q] * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * sq)
                a = feq(u, usq)
                p.append(f[q] - (f[q] - a) / tau + feq(us, ssq) - a)
        else:
            p = _collide64(f, e, w, rho, u, F0, tau)
        f = _stream_walls64(p, e, opp, wm)
        rho, u = _moments64(f, e, None)
        if two:
            low = rho < 0.01
            f = [torch.where(low, x * (0.01 / rho.clamp(min=1e-20)), x) for x in f]
            rho = torch.where(low, 0.01, rho)
        vel = [torch.where(wm, 0.0, v) for v in u]
        if not two:
            c = sum(g)
            post = []
            for q in range(7):
                eu = sum(_E3[q][d] * vel[d] for d in range(3))
                geq = _W7[q] * c * (1 + 3 * eu)
                post.append(torch.where(wm, g[q], g[q] - (g[q] - geq) / _PIPE["tau_tracer"]))
            g = _stream_walls64(post, _E3[:7], opp[:7], wm)
    if two:
        tracer = ((rho - _MP["rho_gas"]) / (_MP["rho_liquid"] - _MP["rho_gas"])).clamp(0, 1)
    else:
        tracer = sum(g)
    return {"f": torch.stack(f, dim=-1), "density": rho, "velocity": torch.stack(vel, dim=-1),
            "tracer": torch.where(wm, 0.0, tracer), "tracer_f": torch.stack(g, dim=-1)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "pipe":
        return _pipe64(case, seed)
    if kind == "ensemble":
        out = []
        for i, (shape, tau, g) in enumerate(_members(case)):
            f, wall, _, _, _ = _flow(case, seed + 17 * i, shape, "channel", "force")
            out.append(_run64(f, wall, {"body_force": np.array([g, 0, 0], dtype=np.float32)},
                              False, tau, case["steps"]))
        return out
    shape = _shape(case)
    f, wall, bi, extra, tau = _flow(case, seed, shape, case["walls"], case["drive"])
    if kind == "gradient":
        force = bi["body_force"]
        if not isinstance(force, torch.Tensor):
            force = torch.as_tensor(force, device=f.device)
        return _gradient64(f, wall, force, tau, case["steps"])
    out = _run64(f, wall, bi, bool(extra), tau, case.get("steps", 1))
    return {**out, "wall_mask": None}
