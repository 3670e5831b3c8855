"""Launch forms of the planned collision and of the host copies at the sizes
where they can go wrong: boxes below, at and above one tile, odd sizes, plans
with and without a lane list and with nothing but one, an odd number of steps
(the tiles run in descending order in the odd ones)."""
import numpy as np
import pytest

from tests.gpu_helpers import rel_l2, rel_max
from virtualfluids_b200 import kernels as K
from virtualfluids_b200.grid import MultipleGridBuilder, SideType, Sphere
from virtualfluids_b200.simulation import BoundaryConditionFactory, Parameter, Simulation

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def grid(nx, ny, nz, sphere=None):
    b = MultipleGridBuilder()
    b.addCoarseGrid(0, 0, 0, nx, ny, nz, 1.0)
    if sphere:
        b.addGeometry(Sphere(*sphere))
    b.setPeriodicBoundaryCondition(sphere is None, sphere is None, sphere is None)
    b.buildGrids()
    for side in (SideType.MX, SideType.PX, SideType.MY, SideType.PY, SideType.MZ, SideType.PZ):
        if sphere:
            b.setVelocityBoundaryCondition(side, 0.0, 0.0, 0.0)
    if sphere:
        b.setNoSlipBoundaryCondition(SideType.GEOMETRY)
    return b.arrays()[0]


def steps_of(g, dtype, kernel, planned, steps, forces=(0.0, 0.0, 0.0)):
    lat = K.DeviceLattice.from_arrays(g)
    rng = np.random.default_rng(3)
    cd = K.compute_dtype(dtype)
    n = len(g["geo"])
    fields = [torch.from_numpy(1e-2 * rng.uniform(-1, 1, n)).to("cuda", cd) for _ in range(4)]
    dist = K.new_distributions(lat, dtype)
    for even in (False, True):
        K.init_equilibrium(dist, lat, *fields, even)
    plan = K.CollisionPlan(dtype, lat) if planned else None
    for t in range(steps):
        K.collision(kernel, dist, lat, 1.7, t % 2 == 0, plan=plan, forces=forces)
    return K.decode(dist), plan.stats() if planned else None


# tolerances of tests/test_gpu_planned.py: FP64 rounding, the FP32 contract, a few units of FP16's rounding
@pytest.mark.parametrize("dtype,tol", [("float64", 1e-12), ("float32", 1e-5), ("float16", 2e-3)])
@pytest.mark.parametrize("kernel", ["K17", "BGK"])
@pytest.mark.parametrize("size,sphere,steps", [((4, 3, 5), None, 3), ((16, 16, 1), None, 2), ((23, 9, 7), None, 5),
                                               ((61, 5, 6), None, 4), ((20, 21, 22), (10.3, 10.1, 11.2, 4.6), 3)])
def test_planned_equals_generic(cuda, dtype, tol, kernel, size, sphere, steps):
    g = grid(*size, sphere=sphere)
    forces = (1e-4, 0.0, -2e-4) if steps == 3 else (0.0, 0.0, 0.0)
    got, stats = steps_of(g, getattr(torch, dtype), kernel, True, steps, forces)
    ref, _ = steps_of(g, getattr(torch, dtype), kernel, False, steps, forces)
    assert stats["bulk_nodes"] + stats["lane_nodes"] == len(g["fluid"])
    assert (rel_max if dtype == "float64" else rel_l2)(got, ref) < tol


@pytest.mark.parametrize("n", [20, 79, 80, 121])
def test_output_copies_equal_plain_copies(cuda, n):
    """The fields of a level below and above the size from which several
    threads copy them (2 MiB in all), into pageable and into pinned arrays."""
    b = MultipleGridBuilder()
    b.addCoarseGrid(0, 0, 0, n - 1, 39, 40, 1.0)
    b.buildGrids()
    b.setVelocityBoundaryCondition(SideType.PZ, 0.05, 0.0, 0.0)
    p = Parameter()
    p.set_viscosity_LB(0.01)
    p.set_storage("fp32")
    sim = Simulation(p, b, BoundaryConditionFactory())
    N = len(sim.levels[0]["geo"])
    rng = np.random.default_rng(n)
    sim.init_level(0, *[1e-3 * rng.uniform(-1, 1, N) for _ in range(4)])
    sim.run(3)
    pinned = [torch.zeros(N, dtype=torch.float32, pin_memory=True).numpy() for _ in range(4)]
    sim.macroscopic(0, out=pinned)
    for _ in range(2):
        for a, ref in zip(sim.macroscopic(0), pinned):
            assert np.array_equal(a, ref)
        out = sim.output(0)
        for a, ref in zip(out["fields"], pinned):
            assert np.array_equal(a, ref)
        assert out["enstrophy"] == sim.enstrophy(0)[0]
    sim.close()
