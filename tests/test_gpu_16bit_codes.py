"""The codes the K17 collision stores in 16 bits, digest for digest.

A 16-bit store keeps the FP32 result's rounding visible: a relaxation x - w x
formed with two roundings instead of one stores another code in one value of
4000 a step (FP16; FX16 one of 70000), and a result that should stay as it is
drifts from then on.  The digests are of the populations after 1 and 4 steps
from integer-made codes (none of the host's arithmetic is in them), on a
periodic box of several tiles with a remainder.
"""
import hashlib

import numpy as np
import pytest

from virtualfluids_b200 import kernels as K
from virtualfluids_b200.grid import MultipleGridBuilder

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# (storage, planned, steps): SHA-256, first 16 digits
DIGESTS = {
    ("float16", True, 1): "7266372c8583137c",
    ("float16", True, 4): "442fa6336fa79708",
    ("float16", False, 1): "a733c02d53838d85",
    ("float16", False, 4): "7bc2ff2b79ea24b6",
    ("bfloat16", True, 1): "ed7811708b1cd735",
    ("bfloat16", True, 4): "9c87899ac53e37b5",
    ("bfloat16", False, 1): "4515237a6b8da759",
    ("bfloat16", False, 4): "9b082423d4dc5d7c",
    ("int16", True, 1): "137a33a1c18d72a9",
    ("int16", True, 4): "2fbcbfb7b7d1ba71",
    ("int16", False, 1): "0e63dab8829441e0",
    ("int16", False, 4): "d797d519aab732ac",
}


def box(nx, ny, nz):
    b = MultipleGridBuilder()
    b.addCoarseGrid(0, 0, 0, nx, ny, nz, 1.0)
    b.setPeriodicBoundaryCondition(True, True, True)
    b.buildGrids()
    return b.arrays()[0]


def start_codes(n, dtype):
    """Pseudo-random stored numbers of n populations, |f - w| < 1e-3 (FX16: 0.016 w)."""
    i = np.arange(1, n + 1, dtype=np.uint64)
    mask = np.uint64(0xffffffff)
    h = (i * np.uint64(2654435761)) & mask
    h = ((h ^ (h >> np.uint64(15))) * np.uint64(2246822519)) & mask
    v = ((h >> np.uint64(8)) % np.uint64(255)).astype(np.int64) - 127
    if dtype == torch.int16:
        return torch.from_numpy((16 * v).astype(np.int16))
    return torch.from_numpy(v / 32.0 if dtype == torch.float16 else v * 2.0 ** -17).to(dtype)


def digest(storage, planned, steps):
    dtype = getattr(torch, storage)
    lat = K.DeviceLattice.from_arrays(box(61, 40, 6))
    dist = start_codes(27 * lat.N, dtype).cuda()
    plan = K.CollisionPlan(dtype, lat) if planned else None
    for t in range(steps):
        K.collision("K17", dist, lat, 1.7, t % 2 == 0, plan=plan)
    return hashlib.sha256(dist.view(torch.int16).cpu().numpy().tobytes()).hexdigest()[:16]


@pytest.mark.parametrize("storage", ["float16", "bfloat16", "int16"])
@pytest.mark.parametrize("planned", [True, False])
@pytest.mark.parametrize("steps", [1, 4])
def test_stored_codes(cuda, storage, planned, steps):
    assert digest(storage, planned, steps) == DIGESTS[storage, planned, steps]
