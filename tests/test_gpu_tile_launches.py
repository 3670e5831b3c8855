"""Launch forms of the planned collision and of the output at the sizes where
they can go wrong: boxes below, at and above one tile, odd sizes, plans with and
without a lane list and with nothing but one, an odd number of steps (the tiles
run in descending order in the odd ones), outputs below and above the number of
blocks that the partial sums' buffer holds at most."""
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


# 256 nodes a block; the output pass runs at most eight blocks an SM, the enstrophy four (B200: 1184 and 592):
# 41 x 43 x 44 nodes (304 blocks), 103 x 43 x 44 (762, between the two), 210 x 43 x 44 (1553, above both)
@pytest.mark.parametrize("n", [39, 101, 208])
@pytest.mark.parametrize("inverse", [True, False])
def test_output_equals_separate_calls(cuda, n, inverse):
    """All values of the output against the separate passes, twice with a step
    between, since the second call finds the first one's partial sums; a level
    without inverse neighbours has no enstrophy section.  The sums to 1e-12 (order
    of summation), counts and fields exactly."""
    b = MultipleGridBuilder()
    b.addCoarseGrid(0, 0, 0, n, 41, 42, 1.0)
    b.buildGrids()
    b.setVelocityBoundaryCondition(SideType.PZ, 0.05, 0.0, 0.0)
    g = dict(b.arrays()[0])
    if not inverse:
        del g["neighborNeg"]
    p = Parameter()
    p.set_viscosity_LB(0.01)
    p.set_storage("fp32")
    sim = Simulation(p, [g], BoundaryConditionFactory())
    N = len(g["geo"])
    rng = np.random.default_rng(n)
    sim.init_level(0, *[np.where(g["geo"] == 19, 1e-3 * rng.uniform(-1, 1, N), 0.0) for _ in range(4)])
    for steps in (3, 1):
        sim.run(steps)
        out = sim.output(0)
        for a, ref in zip(out["fields"], sim.macroscopic(0)):
            assert np.array_equal(a, ref)
        mass, energy, bad = sim.mass_and_energy(0)
        kinetic, kinetic_nodes = sim.kinetic_energy(0)
        enstrophy, enstrophy_nodes = sim.enstrophy(0) if inverse else (0.0, 0)
        assert out["nonfinite"] == bad == 0 and out["fluid_nodes"] == len(g["fluid"])
        assert out["kinetic_energy_nodes"] == kinetic_nodes and out["enstrophy_nodes"] == enstrophy_nodes
        assert (enstrophy_nodes > 0) == inverse and energy > 0
        for got, ref in ((out["mass"], mass), (out["energy"], energy), (out["kinetic_energy"], kinetic),
                         (out["enstrophy"], enstrophy)):
            assert abs(got - ref) <= 1e-12 * max(abs(ref), energy)
    sim.close()
