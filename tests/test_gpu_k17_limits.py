"""The device's reciprocals (an approximation with Newton-Raphson steps) and the
bounds on the limiters, at the ends of the limiters' range: one K17 pass against
the oracle, which divides.  Half of the nodes are at rest, so that their third
moments are exactly zero and a limiter's denominator is the limiter alone.

The oracle's limiter 0 is 1e-30 (FP32 and FP64 alike: the reference divides 0 by
0 at rest); every moment of a node in motion is far above it, so the limited rate
is the full one in both.

Tolerance: that of the node tests on the host (tests/test_k17_limits_host.py),
a few eps of the largest population."""
import numpy as np
import pytest

from oracle.pyoracle import Oracle
from tests.gpu_helpers import rel_max
from virtualfluids_b200 import kernels as K
from virtualfluids_b200.grid import MultipleGridBuilder

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

W = np.array([8 / 27] + [2 / 27] * 6 + [1 / 54] * 12 + [1 / 216] * 8)


@pytest.mark.parametrize("precision,tol", [("f64", 1e-13), ("f32", 2e-6)])
@pytest.mark.parametrize("planned", [True, False])
@pytest.mark.parametrize("limiter", [0.0, 1e-35, 1e-12, 1e15, 1e25, np.inf])
@pytest.mark.parametrize("omega", [0.51, 1.9995])
def test_limiters_at_their_ends(cuda, precision, tol, planned, limiter, omega):
    b = MultipleGridBuilder()
    b.addCoarseGrid(0, 0, 0, 33, 9, 8, 1.0)
    b.setPeriodicBoundaryCondition(True, True, True)
    b.buildGrids()
    g = b.arrays()[0]
    O = Oracle(precision)
    lat = K.DeviceLattice.from_arrays(g)
    N = lat.N
    rng = np.random.default_rng(17)
    f = (rng.uniform(-0.5, 0.5, (27, N)) * W[:, None]).astype(O.real)
    # blocks of rest: a node whose 27 populations all lie in one has no moments
    f[:, (np.arange(N) // (N // 4)) % 2 == 0] = 0
    ref = f.ravel().copy()
    O.collision_k17(ref, N, g["neighborX"], g["neighborY"], g["neighborZ"], g["fluid"], omega,
                    limiters=(max(limiter, 1e-30),) * 3, is_even=True)
    dtype = torch.float64 if precision == "f64" else torch.float32
    dist = torch.from_numpy(f.ravel()).cuda()
    plan = K.CollisionPlan(dtype, lat) if planned else None
    K.collision("K17", dist, lat, omega, True, plan=plan, limiters=(limiter,) * 3)
    got = dist.cpu().numpy()
    assert np.all(np.isfinite(ref)) and np.any(ref == 0)
    assert rel_max(got, ref) < tol
