"""The workloads the framework's speed is measured on.

Each case is one use of the public entry points: the planned collide + stream
passes on periodic boxes (``virtualfluids_b200.kernels``), scheduled time
steps with boundary conditions on one and two levels, the output pass
(``virtualfluids_b200.simulation``), and a gradient through the adjoint time
step (``virtualfluids_b200.adjoint``).  Sizes and parameters are those of the
repository's workloads (cavity 64^3, Taylor-Green 128^3 / 256^3, the
wall-mounted cube, the adjoint channel) or generic ones of the same kind.

``exact`` restates the time step in plain 64-bit torch: the cumulant
collision in full central moments, BGK, the interpolated boundary conditions
and the non-equilibrium pressure outlet, on the sparse index arrays.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from virtualfluids_b200 import kernels as K
from virtualfluids_b200.adjoint import FlowObjective, FlowProblem
from virtualfluids_b200.grid import MultipleGridBuilder, SideType
from virtualfluids_b200.simulation import (BoundaryConditionFactory, NoSlipBC, Parameter, PressureBC, Simulation,
                                           SlipBC)
from virtualfluids_b200.workloads import (adjoint_channel_builder, inlet_entries, inlet_profile, initial_fields,
                                          objective_box, taylor_green_viscosity, wall_mounted_cube)

DTYPES = {"fp64": torch.float64, "fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16,
          "fx16": torch.int16}
BYTES = {"fp64": 8, "fp32": 4, "fp16": 2, "bf16": 2, "fx16": 2, "fx16w": 2}


# --------------------------------------------------------------------- cases --
def listed():
    return [
        # the smallest scheduled simulation: set-up studies and tests, a few launches per step
        {"name": "cavity24_fp32", "kind": "cavity", "nx": 24, "ny": 24, "nz": 24, "storage": "fp32", "steps": 2},
        # the lid-driven cavity of the parity runs, FP64, at its stated size
        {"name": "cavity64_fp64", "kind": "cavity", "nx": 64, "ny": 64, "nz": 64, "storage": "fp64", "steps": 2},
        # a cavity larger than L2: wall lists beside a memory-bound collision, ragged sizes
        {"name": "cavity_ragged_fp32", "kind": "cavity", "nx": 161, "ny": 150, "nz": 173, "storage": "fp32", "steps": 2},
        # Taylor-Green at its smallest stated size, FP64: the parity precision of the collision
        {"name": "box128_k17_fp64", "kind": "box", "nx": 128, "ny": 128, "nz": 128, "storage": "fp64", "kernel": "K17",
         "steps": 2},
        # Taylor-Green 256^3 FP32, the plain form: the bandwidth benchmark's kernel
        {"name": "box256_k17_fp32", "kind": "box", "nx": 256, "ny": 256, "nz": 256, "storage": "fp32", "kernel": "K17",
         "steps": 2},
        # the BGK variant on an odd-sized periodic box
        {"name": "box_ragged_bgk_fp32", "kind": "box", "nx": 219, "ny": 187, "nz": 133, "storage": "fp32",
         "kernel": "BGK", "steps": 2},
        # the precision form: half storage of the shifted populations
        {"name": "box192_k17_fp16", "kind": "box", "nx": 192, "ny": 192, "nz": 192, "storage": "fp16", "kernel": "K17",
         "steps": 2},
        # the precision form's fixed-point storage, its velocity read out after four steps
        {"name": "box320_k17_fx16", "kind": "box", "nx": 320, "ny": 320, "nz": 320, "storage": "fx16", "kernel": "K17",
         "steps": 4},
        # the wall-mounted cube on two levels at its stated size: BC lists, refinement interface, schedule
        {"name": "cube_two_level_fp32", "kind": "cube", "nx": 256, "ny": 96, "nz": 96, "storage": "fp32", "steps": 2},
        # the same in the precision form
        {"name": "cube_two_level_fp16", "kind": "cube", "nx": 256, "ny": 96, "nz": 96, "storage": "fp16", "steps": 2},
        # gradient of a downstream objective: checkpointed forward steps and the adjoint steps backwards
        {"name": "adjoint_channel_fp32", "kind": "adjoint", "nx": 128, "ny": 64, "nz": 64, "storage": "fp32",
         "steps": 128, "interval": 32},
        # the output of a simulation: fields to the host with the FP64 sums and the analyzers
        {"name": "output_channel_fp32", "kind": "output", "nx": 160, "ny": 96, "nz": 97, "storage": "fp32", "steps": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "box", "box", "cavity", "cavity", "cube", "adjoint", "output"])
    if kind == "box":
        storage = rng.choice(["fp64", "fp32", "fp32", "fp16", "bf16", "fx16"])
        top = 224 if storage == "fp64" else 270
        return {"kind": "box", "nx": _log(rng, 20, top), "ny": _log(rng, 20, top), "nz": _log(rng, 20, top),
                "storage": storage, "kernel": rng.choice(["K17", "K17", "K17", "BGK"]),
                "steps": 4 if storage == "fx16" else 2}
    if kind == "cavity":
        return {"kind": "cavity", "nx": _log(rng, 16, 170), "ny": _log(rng, 16, 170), "nz": _log(rng, 16, 170),
                "storage": rng.choice(["fp64", "fp32", "fp32", "fp16"]), "steps": 2 * rng.randint(1, 3)}
    if kind == "cube":
        return {"kind": "cube", "nx": rng.randint(152, 256), "ny": rng.randint(88, 108), "nz": rng.randint(76, 104),
                "storage": rng.choice(["fp64", "fp32", "fp16", "bf16"]), "steps": 2}
    if kind == "adjoint":
        return {"kind": "adjoint", "nx": rng.randint(100, 128), "ny": rng.randint(30, 64), "nz": rng.randint(30, 64),
                "storage": rng.choice(["fp64", "fp32", "fp32"]), "steps": rng.randint(90, 128),
                "interval": rng.choice([16, 32, 64, 128])}
    return {"kind": "output", "nx": _log(rng, 40, 160), "ny": _log(rng, 40, 100), "nz": _log(rng, 40, 100),
            "storage": rng.choice(["fp64", "fp32", "fp16"]), "steps": 2}


# ------------------------------------------------------------ periodic boxes --
def _box_arrays(nx, ny, nz):
    """Index arrays of a periodic nx x ny x nz box in the builder's layout
    (one layer of stoppers around the fluid, node 0 a dummy), on the GPU."""
    dev = _device()
    px, py, pz = nx + 2, ny + 2, nz + 2
    N = px * py * pz + 1
    k = torch.arange(px * py * pz, device=dev, dtype=torch.int32)
    x, y, z = k % px, (k // px) % py, k // (px * py)
    fluid = (x >= 1) & (x <= nx) & (y >= 1) & (y <= ny) & (z >= 1) & (z <= nz)

    def neighbour(pos, n, stride):
        nxt = torch.where(fluid & (pos == n), k - (n - 1) * stride, k + stride) + 1
        nxt = torch.where(pos == n + 1, torch.zeros_like(nxt), nxt)
        return torch.cat([torch.zeros(1, device=dev, dtype=torch.int32), nxt]).contiguous()

    geo = torch.full((N,), 16, device=dev, dtype=torch.int32)
    geo[1:][fluid] = 19
    return {"N": N, "nX": neighbour(x, nx, 1), "nY": neighbour(y, ny, px), "nZ": neighbour(z, nz, px * py), "geo": geo,
            "fluid": (torch.nonzero(fluid).flatten() + 1).to(torch.int32)}


def _box_omega(case):
    return 1.0 / (3.0 * taylor_green_viscosity(min(case["nx"], case["ny"], case["nz"])) + 0.5)


def _box_fields(case, seed, dtype):
    """Taylor-Green with seeded noise of 1e-3 u0 on the velocity (zero outside the fluid)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    u0 = 0.05
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def axis(n):
        return (2.0 * math.pi / n) * (torch.arange(n, device="cuda", dtype=torch.float32) - (n - 1) / 2.0)

    X, Y, Z = axis(nx)[None, None, :], axis(ny)[None, :, None], axis(nz)[:, None, None]
    shape = (nz, ny, nx)
    rho = 3.0 * u0 * u0 / 16.0 * (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2.0)
    vel = [u0 * torch.sin(X) * torch.cos(Y) * torch.cos(Z), -u0 * torch.cos(X) * torch.sin(Y) * torch.cos(Z),
           torch.zeros(shape, device="cuda")]
    fields = [rho] + [v + 1e-3 * u0 * (2.0 * torch.rand(shape, generator=gen, device="cuda") - 1.0) for v in vel]
    out = []
    for f in fields:
        a = torch.zeros((nz + 2, ny + 2, nx + 2), device="cuda", dtype=dtype)
        a[1:-1, 1:-1, 1:-1] = f.to(dtype)
        out.append(torch.cat([torch.zeros(1, device="cuda", dtype=dtype), a.reshape(-1)]))
    return out


def _prepare_box(case, seed):
    a = _box_arrays(case["nx"], case["ny"], case["nz"])
    dtype = DTYPES[case["storage"]]
    lat = K.DeviceLattice(a["N"], a["nX"], a["nY"], a["nZ"], a["geo"], a["fluid"])
    dist = K.new_distributions(lat, dtype)
    fields = _box_fields(case, seed, K.compute_dtype(dtype))
    for even in (False, True):
        K.init_equilibrium(dist, lat, *fields, even)
    return {"case": case, "lat": lat, "dist": dist, "plan": K.CollisionPlan(dtype, lat), "omega": _box_omega(case)}


def _run_box(s):
    case, dist = s["case"], s["dist"]
    for t in range(case["steps"]):
        K.collision(case["kernel"], dist, s["lat"], s["omega"], t % 2 == 0, plan=s["plan"])
    if case["storage"] == "fx16":
        # codes of a fixed-point store: the velocity is what such a run is read out by
        return K.macroscopic(dist, s["lat"], True)
    return dist


# --------------------------------------------------------------- simulations --
@functools.lru_cache(maxsize=4)
def _cavity_levels(nx, ny, nz):
    b = MultipleGridBuilder()
    b.addCoarseGrid(0, 0, 0, nx - 1, ny - 1, nz - 1, 1.0)
    b.buildGrids()
    for side in (SideType.MX, SideType.PX, SideType.MY, SideType.PY, SideType.MZ):
        b.setNoSlipBoundaryCondition(side)
    b.setVelocityBoundaryCondition(SideType.PZ, 0.05, 0.0, 0.0)
    return b.arrays()


@functools.lru_cache(maxsize=4)
def _output_levels(nx, ny, nz):
    """A channel with an inlet, an outlet, walls, and a solid block on the floor."""
    b = MultipleGridBuilder()
    b.addCoarseGrid(0, 0, 0, nx, ny, nz, 1.0)
    b.addGeometry((nx // 4, ny // 3, 0, nx // 4 + ny // 4, ny // 3 + ny // 4, nz // 4))
    b.buildGrids()
    b.setVelocityBoundaryCondition(SideType.MX, 0.04, 0.0, 0.0)
    b.setPressureBoundaryCondition(SideType.PX, 0.0)
    for side in (SideType.MY, SideType.PY, SideType.MZ, SideType.PZ):
        b.setNoSlipBoundaryCondition(side)
    b.setNoSlipBoundaryCondition(SideType.GEOMETRY)
    return b.arrays()


@functools.lru_cache(maxsize=2)
def _cube_levels(nx, ny, nz):
    return wall_mounted_cube(coarse=(nx, ny, nz), box=(48, ny // 2 - 24, 0, 128, ny // 2 + 24, 40), noise=0.0)


@functools.lru_cache(maxsize=2)
def _adjoint_levels(nx, ny, nz):
    return adjoint_channel_builder(nx, ny, nz, (40, ny // 2 - 6, nz // 2 - 6, 52, ny // 2 + 6, nz // 2 + 6)).arrays()


def _levels(case):
    make = {"cavity": _cavity_levels, "output": _output_levels, "cube": _cube_levels, "adjoint": _adjoint_levels}
    return make[case["kind"]](case["nx"], case["ny"], case["nz"])


def _viscosity(case):
    if case["kind"] == "cavity":
        return 0.05 * min(case["nx"], case["ny"], case["nz"]) / 1000.0  # Re = 1000 on the shortest side
    return {"cube": 0.04 * 16 / 2000.0, "adjoint": 0.02, "output": 0.01}[case["kind"]]


def _initial(case, g, seed, level=0):
    """(drho, vx, vy, vz) host arrays: the flow at rest (cavity), or the channel's stream, with seeded noise."""
    rng = np.random.default_rng([seed, level])
    n = len(g["geo"])
    u = 0.0 if case["kind"] == "cavity" else 0.04
    fields = [1e-4 * rng.uniform(-1, 1, n), u + 1e-3 * rng.uniform(-1, 1, n), 1e-3 * rng.uniform(-1, 1, n),
              1e-3 * rng.uniform(-1, 1, n)]
    for f in fields:
        f[g["geo"] != 19] = 0.0
    return fields


def _factory(case):
    bc = BoundaryConditionFactory()
    if case["kind"] != "cavity":
        bc.set_geometry_boundary_condition(NoSlipBC.NoSlipInterpolatedCompressible)
        bc.set_pressure_boundary_condition(PressureBC.PressureNonEquilibriumCompressible)
    if case["kind"] == "cube":
        bc.set_slip_boundary_condition(SlipBC.SlipCompressible)
    return bc


def _simulation(case, levels):
    p = Parameter()
    p.set_viscosity_LB(_viscosity(case))
    p.set_storage(case["storage"])
    if case["kind"] == "adjoint":
        p.set_forcing(1e-6, 0.0, 0.0)
    return Simulation(p, levels, _factory(case))


class _DeviceArray:
    def __init__(self, pointer, count, typestr):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (pointer, False), "version": 3}


def _populations(sim, level, storage):
    """The level's populations as a tensor (the simulation's own buffer, which
    the tensor keeps alive)."""
    pointer, n, _, _ = sim.level_state(level)
    t = torch.as_tensor(_DeviceArray(pointer, 27 * n, {"fp64": "<f8", "fp32": "<f4"}.get(storage, "<i2")),
                        device="cuda")
    t = t.view(torch.bfloat16) if storage == "bf16" else t.view(torch.float16) if storage == "fp16" else t
    t.simulation = sim
    return t


def _noisy_inlet(levels, seed):
    """The cube's levels with +-1% of noise on the inlet's velocities."""
    rng = np.random.default_rng(seed)
    out = []
    for g in levels:
        g = dict(g)
        vx = g["velocity.vx"].copy()
        inflow = vx != 0
        vx[inflow] *= 1.0 + rng.uniform(-0.01, 0.01, int(inflow.sum()))
        g["velocity.vx"] = vx
        out.append(g)
    return out


def _prepare_simulation(case, seed):
    levels = _levels(case)
    if case["kind"] == "cube":
        levels = _noisy_inlet(levels, seed)
    sim = _simulation(case, levels)
    for lvl, g in enumerate(levels):
        sim.init_level(lvl, *_initial(case, g, seed, lvl))
    if case["kind"] == "output":
        sim.run(case["steps"])
        return {"case": case, "sim": sim}
    return {"case": case, "sim": sim, "out": [_populations(sim, lvl, case["storage"]) for lvl in range(len(levels))]}


def _run_simulation(s):
    s["sim"].run(s["case"]["steps"])
    return s["out"]


def _run_output(s):
    r = s["sim"].output(0)
    return {"fields": r["fields"], "sums": np.array([r["mass"], r["energy"], r["kinetic_energy"], r["enstrophy"]]),
            "counts": np.array([r["nonfinite"], r["kinetic_energy_nodes"], r["enstrophy_nodes"], r["fluid_nodes"]])}


# ------------------------------------------------------------------- adjoint --
def _objective_nodes(case, g):
    ny, nz = case["ny"], case["nz"]
    return objective_box(g, 80, 96, ny // 2 - 8, ny // 2 + 8, nz // 2 - 8, nz // 2 + 8)


def _prepare_adjoint(case, seed):
    levels = _levels(case)
    sim = _simulation(case, levels)
    g = sim.levels[0]
    nodes, weights = _objective_nodes(case, g)
    problem = FlowProblem(sim, inlet_entries(g), initial_fields(g), case["steps"], case["interval"], nodes,
                          (weights, None, None))
    return {"case": case, "sim": sim, "problem": problem,
            "profile": torch.from_numpy(inlet_profile(g, seed=seed)).requires_grad_(),
            "force": torch.tensor([1e-6, 0.0, 0.0], dtype=torch.float64, requires_grad=True),
            "state": _populations(sim, 0, case["storage"])}


def _run_adjoint(s):
    s["profile"].grad = s["force"].grad = None
    J = FlowObjective.apply(s["profile"], s["force"], s["problem"])
    J.backward()
    return {"J": J.detach(), "profile": s["profile"].grad, "force": s["force"].grad, "state": s["state"]}


# ------------------------------------------------------------------ contract --
def prepare(case, seed):
    if case["kind"] == "box":
        return _prepare_box(case, seed)
    if case["kind"] == "adjoint":
        return _prepare_adjoint(case, seed)
    return _prepare_simulation(case, seed)


def run(state):
    return {"box": _run_box, "cavity": _run_simulation, "cube": _run_simulation, "output": _run_output,
            "adjoint": _run_adjoint}[state["case"]["kind"]](state)


def _nodes(case):
    """Node updates of one step."""
    if case["kind"] == "box":
        return case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "cube":
        # the coarse level without the refined box's inside, and the two substeps of the fine level
        # (a box of 80 x 48 x 40 coarse nodes and its overlap, the same for every coarse size)
        return (case["nx"] - 1) * case["ny"] * (case["nz"] - 1) - 223_917 + 2 * 1_921_548
    return (case["nx"] - 1) * (case["ny"] - 1) * (case["nz"] - 1)


def work(case):
    s, n, steps = BYTES[case["storage"]], _nodes(case), case["steps"]
    step = 2 * 27 * s  # every population read and written once
    r = 8 if case["storage"] == "fp64" else 4
    if case["kind"] == "output":
        # the populations read once, four fields written and taken to the host
        return {"bytes": n * (27 * s + 4 * r), "flops": 150 * n}
    if case["kind"] == "adjoint":
        # forward steps; backwards the adjoint state read and written, the pre-collision values read
        return {"bytes": n * steps * (step + 3 * 27 * s), "flops": 2500 * n * steps}
    extra = n * (27 * s + 4 * r) if case["storage"] == "fx16" else 0
    flops = 250 if case.get("kernel") == "BGK" else 700
    return {"bytes": n * steps * step + extra, "flops": flops * n * steps}


def tolerance(case):
    """About four times what the two collision paths (planned and index-chain
    kernels, whose sums run in another order) or the 64-bit restatement show."""
    s = case["storage"]
    if case["kind"] == "adjoint":
        return {"rel": 2e-12, "max": 2e-10} if s == "fp64" else {"rel": 1e-5, "max": 1e-3}
    if s == "fp64":
        return {"rel": 6e-13, "max": 4e-11}
    if s == "fp32":
        return {"rel": 1e-5, "max": 4e-4} if case["kind"] == "output" else {"rel": 2e-6, "max": 6e-5}
    if s == "fx16":
        return {"rel": 7e-3, "max": 0.17}  # of the z velocity, which is little more than noise
    return {"rel": 1e-4, "max": 0.02} if s == "fp16" else {"rel": 3e-4, "max": 0.1}


# --------------------------------------------------- the step in 64-bit torch --
CX = [0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1]
CY = [0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1, 1, 1, -1, -1, 1, 1, -1, -1]
CZ = [0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1, 1, 1, 1, 1, -1, -1, -1, -1]
C = list(zip(CX, CY, CZ))
INV = [C.index((-x, -y, -z)) for x, y, z in C]
W = [[8 / 27, 2 / 27, 1 / 54, 1 / 216][abs(x) + abs(y) + abs(z)] for x, y, z in C]
LOC = [(x < 0) + 2 * (y < 0) + 4 * (z < 0) for x, y, z in C]


def _along(d, u):
    return sum(c * v for c, v in zip(C[d], u) if c) if d else 0.0 * u[0]


def _macros(f):
    rho = sum(f) + 1.0
    return rho, [sum(C[d][a] * f[d] for d in range(27) if C[d][a]) / rho for a in range(3)]


def _bgk(f, omega, force):
    rho, u = _macros(f)
    usq = 1.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    out = []
    for d in range(27):
        cu = _along(d, u)
        out.append(f[d] + omega * (W[d] * (rho - 1.0 + rho * (3.0 * cu + 4.5 * cu * cu - usq)) - f[d]))
    return out


def _k17(f, omega, force):
    """The compressible cumulant collision (third-order limiters 0.01, fourth-order
    optimised equilibrium) in full central moments."""
    limiter = 0.01
    rho, u = _macros(f)
    v = [u[a] + force[a] for a in range(3)]
    # central moments, axis by axis
    m = {C[d]: f[d] + W[d] for d in range(27)}
    for a in range(3):
        new = {}
        for key in m:
            if key[a] != 0:
                continue

            def at(c):
                return m[key[:a] + (c,) + key[a + 1:]]

            lo, mid, hi = at(-1), at(0), at(1)
            s, diff, sq = lo + mid + hi, hi - lo, hi + lo
            # entries -1 / 0 / 1 of the axis now stand for the orders 0 / 1 / 2
            new[key[:a] + (-1,) + key[a + 1:]] = s
            new[key] = diff - v[a] * s
            new[key[:a] + (1,) + key[a + 1:]] = sq - 2.0 * v[a] * diff + v[a] * v[a] * s
        m = new
    k = {(x + 1, y + 1, z + 1): val for (x, y, z), val in m.items()}
    o = omega
    xyy_p = 8.0 * (o - 2.0) * (1.0 + 2.0 * o) / (-8.0 - 14.0 * o + 7.0 * o * o)
    xyy_m = 8.0 * (o - 2.0) * (4.0 * o - 7.0) / (56.0 - 50.0 * o + 9.0 * o * o)
    xyz = 24.0 * (o - 2.0) * (-2.0 - 7.0 * o + 3.0 * o * o) / (48.0 + 152.0 * o - 130.0 * o * o + 29.0 * o ** 3)
    A = (4.0 + 2.0 * o - 3.0 * o * o) / (2.0 - 7.0 * o + 5.0 * o * o)
    B = (4.0 + 28.0 * o - 14.0 * o * o) / (6.0 - 21.0 * o + 15.0 * o * o)
    tau = 1.0 / o - 0.5

    def limited(x, rate):
        w = rate + (1.0 - rate) * torch.abs(x) / (torch.abs(x) + limiter)
        return x - w * x

    # velocity gradients and second order
    trace = k[2, 0, 0] + k[0, 2, 0] + k[0, 0, 2]
    xy, xz = k[2, 0, 0] - k[0, 2, 0], k[2, 0, 0] - k[0, 0, 2]
    dx = -0.5 * o * (xy + xz) + 0.5 * (rho - trace)
    dy = dx + 1.5 * o * xy
    dz = dx + 1.5 * o * xz
    gxy, gxz, gyz = -3.0 * o * k[1, 1, 0], -3.0 * o * k[1, 0, 1], -3.0 * o * k[0, 1, 1]
    x2, y2, z2 = v[0] ** 2, v[1] ** 2, v[2] ** 2
    trace = rho - 1.5 * (x2 * dx + y2 * dy + z2 * dz)
    xy = (1.0 - o) * xy - 3.0 * (1.0 - 0.5 * o) * (x2 * dx - y2 * dy)
    xz = (1.0 - o) * xz - 3.0 * (1.0 - 0.5 * o) * (x2 * dx - z2 * dz)
    n = {(0, 0, 0): rho}
    n[2, 0, 0] = (trace + xy + xz) / 3.0
    n[0, 2, 0] = n[2, 0, 0] - xy
    n[0, 0, 2] = n[2, 0, 0] - xz
    for key in ((1, 1, 0), (1, 0, 1), (0, 1, 1)):
        n[key] = (1.0 - o) * k[key]
    # third order
    n[1, 1, 1] = limited(k[1, 1, 1], xyz)
    for p, q in (((2, 1, 0), (0, 1, 2)), ((2, 0, 1), (0, 2, 1)), ((1, 2, 0), (1, 0, 2))):
        plus, minus = limited(k[p] + k[q], xyy_p), limited(k[p] - k[q], xyy_m)
        n[p], n[q] = 0.5 * (plus + minus), 0.5 * (plus - minus)
    # fourth order
    n[2, 2, 0] = (n[2, 0, 0] * n[0, 2, 0] + 2.0 * n[1, 1, 0] ** 2) / rho - tau * 2.0 / 3.0 * A * (dx + dy)
    n[2, 0, 2] = (n[2, 0, 0] * n[0, 0, 2] + 2.0 * n[1, 0, 1] ** 2) / rho - tau * 2.0 / 3.0 * A * (dx + dz)
    n[0, 2, 2] = (n[0, 2, 0] * n[0, 0, 2] + 2.0 * n[0, 1, 1] ** 2) / rho - tau * 2.0 / 3.0 * A * (dy + dz)
    n[2, 1, 1] = (n[2, 0, 0] * n[0, 1, 1] + 2.0 * n[1, 1, 0] * n[1, 0, 1]) / rho - tau / 3.0 * B * gyz
    n[1, 2, 1] = (n[0, 2, 0] * n[1, 0, 1] + 2.0 * n[1, 1, 0] * n[0, 1, 1]) / rho - tau / 3.0 * B * gxz
    n[1, 1, 2] = (n[0, 0, 2] * n[1, 1, 0] + 2.0 * n[1, 0, 1] * n[0, 1, 1]) / rho - tau / 3.0 * B * gxy
    # fifth and sixth order: cumulants zero
    n[1, 2, 2] = (n[0, 0, 2] * n[1, 2, 0] + n[0, 2, 0] * n[1, 0, 2] + 4.0 * n[0, 1, 1] * n[1, 1, 1] +
                  2.0 * (n[1, 0, 1] * n[0, 2, 1] + n[1, 1, 0] * n[0, 1, 2])) / rho
    n[2, 1, 2] = (n[0, 0, 2] * n[2, 1, 0] + n[2, 0, 0] * n[0, 1, 2] + 4.0 * n[1, 0, 1] * n[1, 1, 1] +
                  2.0 * (n[0, 1, 1] * n[2, 0, 1] + n[1, 1, 0] * n[1, 0, 2])) / rho
    n[2, 2, 1] = (n[2, 0, 0] * n[0, 2, 1] + n[0, 2, 0] * n[2, 0, 1] + 4.0 * n[1, 1, 0] * n[1, 1, 1] +
                  2.0 * (n[1, 0, 1] * n[1, 2, 0] + n[0, 1, 1] * n[2, 1, 0])) / rho
    n[2, 2, 2] = (4.0 * n[1, 1, 1] ** 2 + n[2, 0, 0] * n[0, 2, 2] + n[0, 2, 0] * n[2, 0, 2] + n[0, 0, 2] * n[2, 2, 0] +
                  4.0 * (n[0, 1, 1] * n[2, 1, 1] + n[1, 0, 1] * n[1, 2, 1] + n[1, 1, 0] * n[1, 1, 2]) +
                  2.0 * (n[1, 2, 0] * n[1, 0, 2] + n[2, 1, 0] * n[0, 1, 2] + n[2, 0, 1] * n[0, 2, 1])) / rho - \
                 (16.0 * n[1, 1, 0] * n[1, 0, 1] * n[0, 1, 1] +
                  4.0 * (n[1, 0, 1] ** 2 * n[0, 2, 0] + n[0, 1, 1] ** 2 * n[2, 0, 0] + n[1, 1, 0] ** 2 * n[0, 0, 2]) +
                  2.0 * n[2, 0, 0] * n[0, 2, 0] * n[0, 0, 2]) / rho ** 2
    # the force turns the first moments' sign
    n[1, 0, 0], n[0, 1, 0], n[0, 0, 1] = -k[1, 0, 0], -k[0, 1, 0], -k[0, 0, 1]
    # back to populations, axis by axis
    m = n
    for a in range(3):
        new = {}
        for key in m:
            if key[a] != 0:
                continue

            def at(c):
                return m[key[:a] + (c,) + key[a + 1:]]

            r0, r1 = at(0), at(1) + v[a] * at(0)
            r2 = at(2) + 2.0 * v[a] * at(1) + v[a] * v[a] * at(0)
            new[key] = 0.5 * (r2 - r1)
            new[key[:a] + (1,) + key[a + 1:]] = r0 - r2
            new[key[:a] + (2,) + key[a + 1:]] = 0.5 * (r2 + r1)
        m = new
    return [m[C[d][0] + 1, C[d][1] + 1, C[d][2] + 1] - W[d] for d in range(27)]


class _Lattice:
    """One level's flat population tensor D[27 N] and its index arrays (the twisted in-place views)."""

    def __init__(self, N, nX, nY, nZ, fluid, omega, device):
        self.N, self.omega, self.device = N, omega, device
        self.nb = [torch.as_tensor(np.ascontiguousarray(a).view(np.int32) if isinstance(a, np.ndarray) else a,
                                   device=device).long() for a in (nX, nY, nZ)]
        self.fluid = self.index(fluid)

    def index(self, a):
        if isinstance(a, np.ndarray):
            a = torch.from_numpy(np.ascontiguousarray(a).view(np.int32))
        return a.to(self.device).long()

    def locations(self, k):
        nX, nY, nZ = self.nb
        x, y = nX[k], nY[k]
        xy = nY[x]
        return [k, x, y, xy, nZ[k], nZ[x], nZ[y], nZ[xy]]

    def cells(self, L, d, even):
        return (d if even else INV[d]) * self.N + L[LOC[d]]

    def collide(self, D, even, operator, force, chunk=1 << 22):
        if D.requires_grad or torch.is_grad_enabled():
            L = self.locations(self.fluid)
            idx = [self.cells(L, d, even) for d in range(27)]
            f = operator([D[i] for i in idx], self.omega, force)
            return D.index_put((torch.cat(idx),), torch.cat([f[INV[d]] for d in range(27)]))
        for part in self.fluid.split(chunk):
            L = self.locations(part)
            idx = [self.cells(L, d, even) for d in range(27)]
            f = operator([D[i] for i in idx], self.omega, force)
            for d in range(27):
                D[idx[d]] = f[INV[d]]
        return D

    def read(self, D, k, even):
        L = self.locations(k)
        return [D[self.cells(L, d, even)] for d in range(27)]

    def wall(self, D, k, q, U, even):
        """Interpolated bounce-back with the wall velocity U (None: at rest)."""
        L = self.locations(k)
        g = [D[self.cells(L, INV[d], even)] for d in range(27)]
        rho, u = _macros(g)
        usq = 1.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2) * rho
        where, what = [], []
        for d in range(1, 27):
            sel = torch.nonzero((q[d] >= 0) & (q[d] <= 1)).flatten()
            if sel.numel() == 0:
                continue
            e, qd = INV[d], q[d][sel]
            a, b = g[d][sel], g[e][sel]
            cu = _along(d, [c[sel] for c in u])
            feq = W[d] * (rho[sel] - 1.0 + 4.5 * cu * cu * rho[sel] - usq[sel])
            value = 0.5 * (1.0 - qd) / (1.0 + qd) * (a - b + (a + b - 2.0 * feq * self.omega) / (1.0 - self.omega))
            moving = 6.0 * W[d] * _along(d, [c[sel] for c in U]) if U is not None else 0.0
            where.append(self.cells(L, e, not even)[sel])
            what.append(value + (qd * (a + b) - moving) / (1.0 + qd))
        return D.index_put((torch.cat(where),), torch.cat(what)) if where else D

    def outlet(self, D, k, kN, rho_bc, direction, even):
        """The neighbour's populations with their equilibrium moved to the prescribed density."""
        L = self.locations(k)
        f = self.read(D, kN, even)
        rho, u = _macros(f)
        usq = 1.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
        axis = next(a for a in range(3) if C[direction][a])
        where, what = [], []
        for d in range(27):
            if C[d][axis] == C[direction][axis]:
                continue
            cu = _along(d, u)
            shape = 1.0 + 3.0 * cu + 4.5 * cu * cu - usq
            where.append(self.cells(L, d, even))
            what.append(f[d] + W[d] * (rho_bc + 1.0 - rho) * shape)
        return D.index_put((torch.cat(where),), torch.cat(what))


def _equilibrium(rho, u):
    usq = 1.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    out = []
    for d in range(27):
        cu = _along(d, u)
        out.append(W[d] * (rho + (1.0 + rho) * (3.0 * cu + 4.5 * cu * cu - usq)))
    return out


def _start(lat, geo, fields, storage):
    """Populations of the initial fields, in the values that the storage holds, through both views."""
    D = torch.zeros(27 * lat.N, dtype=torch.float64, device=lat.device)
    r = torch.float64 if storage == "fp64" else torch.float32
    fields = [f.to(r).double() for f in fields]
    nodes = torch.nonzero((geo != 15) & (geo != 16)).flatten()
    for even in (False, True):
        for part in nodes.split(1 << 22):
            L = lat.locations(part)
            f = _equilibrium(fields[0][part], [c[part] for c in fields[1:]])
            for d in range(27):
                D[lat.cells(L, d, even)] = f[d]
    return D


def _fields_of(lat, D, geo, even):
    out = [torch.zeros(lat.N, dtype=torch.float64, device=lat.device) for _ in range(4)]
    for part in torch.nonzero((geo != 15) & (geo != 16)).flatten().split(1 << 22):
        rho, u = _macros(lat.read(D, part, even))
        for o, value in zip(out, [rho - 1.0] + u):
            o[part] = value
    return out


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _level(case, g, level=0):
    omega = 1.0 / (3.0 * _viscosity(case) * 2.0 ** level + 0.5)
    lat = _Lattice(len(g["geo"]), g["neighborX"], g["neighborY"], g["neighborZ"], g["fluid"], omega, _device())
    return lat, lat.index(g["geo"])


def _reals(a, case, dev):
    t = torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(dev)
    return t if case["storage"] == "fp64" else t.float().double()


def _schedule(case, g, lat, D, steps, velocity, force, each=lambda f, *a: f(*a)):
    """`steps` single-level steps: collision, velocity and geometry lists, swap, outlet."""
    dev = lat.device
    lists = []
    for name in ("velocity", "geometry"):
        k = lat.index(g[f"{name}.k"])
        if k.numel() and (name == "velocity" or case["kind"] != "cavity"):
            lists.append((k, _reals(g[f"{name}.q"], case, dev).reshape(27, -1), velocity if name == "velocity" else None))
    outlet = None
    if case["kind"] != "cavity":
        outlet = (lat.index(g["pressure0.k"]), lat.index(g["pressure0.kN"]), _reals(g["pressure0.rho"], case, dev),
                  int(g["pressure0.dir"][0]))

    def step(D, even):
        D = lat.collide(D, even, _k17, force)
        for k, q, U in lists:
            D = lat.wall(D, k, q, U, even)
        return D if outlet is None else lat.outlet(D, *outlet, not even)

    for t in range(steps):
        D = each(step, D, t % 2 == 0)
    return D


def _velocity(case, g, dev):
    return [_reals(g[f"velocity.{c}"], case, dev) for c in ("vx", "vy", "vz")]


def _exact_box(case, seed):
    a = _box_arrays(case["nx"], case["ny"], case["nz"])
    lat = _Lattice(a["N"], a["nX"], a["nY"], a["nZ"], a["fluid"], _box_omega(case), "cuda")
    real = torch.float64 if case["storage"] == "fp64" else torch.float32
    D = _start(lat, a["geo"], _box_fields(case, seed, real), case["storage"])
    operator = _k17 if case["kernel"] == "K17" else _bgk
    for t in range(case["steps"]):
        D = lat.collide(D, t % 2 == 0, operator, (0.0, 0.0, 0.0))
    if case["storage"] == "fx16":
        return _fields_of(lat, D, a["geo"], True)
    return D * 4096.0 if case["storage"] == "fp16" else D


def _exact_simulation(case, seed):
    g = _levels(case)[0]
    lat, geo = _level(case, g)
    fields = [torch.from_numpy(f).to(lat.device) for f in _initial(case, g, seed)]
    D = _start(lat, geo, fields, case["storage"])
    D = _schedule(case, g, lat, D, case["steps"], _velocity(case, g, lat.device), (0.0, 0.0, 0.0))
    if case["kind"] == "output":
        # the sums and the enstrophy's stencils depend on the analyzers' node sets: the fields only
        return {"fields": _fields_of(lat, D, geo, case["steps"] % 2 == 0), "sums": None, "counts": None}
    return [D * 4096.0 if case["storage"] == "fp16" else D]


def _exact_adjoint(case, seed):
    g = _levels(case)[0]
    lat, geo = _level(case, g)
    dev = lat.device
    fields = [torch.from_numpy(f).to(dev) for f in initial_fields(g)]
    with torch.no_grad():
        D = _start(lat, geo, fields, case["storage"])
        base = _velocity(case, g, dev)
    profile = torch.from_numpy(inlet_profile(g, seed=seed)).to(dev).requires_grad_()
    force = torch.tensor([1e-6, 0.0, 0.0], dtype=torch.float64, device=dev, requires_grad=True)
    with torch.enable_grad():
        at = torch.from_numpy(inlet_entries(g)).to(dev)
        vx = base[0].index_put((at,), profile)

        def each(step, D, even):
            return checkpoint(step, D, even, use_reentrant=False)

        D = _schedule(case, g, lat, D, case["steps"], [vx, base[1], base[2]], [0.5 * force[a] for a in range(3)], each)
        nodes, weights = _objective_nodes(case, g)
        _, u = _macros(lat.read(D, lat.index(nodes), case["steps"] % 2 == 0))
        J = (torch.from_numpy(weights).to(dev) * u[0]).sum()
        J.backward()
    return {"J": J.detach(), "profile": profile.grad, "force": force.grad, "state": D.detach()}


def exact(case, seed):
    if case["kind"] == "cube":
        return None  # two levels to their interpolation: no statement short enough to stand here
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    with torch.no_grad():
        return _exact_box(case, seed) if case["kind"] == "box" else _exact_simulation(case, seed)
