"""The K17 operator at the ends of its inputs, on the host, against the oracle:
limiters that switch the limiting off (large, beyond the bound the library
clamps at), force zero and not, omega near its ends.

Tolerance: the operator's 470 operations on populations of at most 0.02, each
rounded to eps / 2 of intermediate values no larger than 1: a few eps of the
largest population (FP64 1e-13, FP32 2e-6 as in the other node tests)."""
import numpy as np
import pytest

from oracle.pyoracle import Oracle
from tests.test_collision_math_host import lib_node
from virtualfluids_b200 import _lib

W = np.array([8 / 27] + [2 / 27] * 6 + [1 / 54] * 12 + [1 / 216] * 8)


@pytest.mark.parametrize("precision,tol", [("f64", 1e-13), ("f32", 2e-6)])
@pytest.mark.parametrize("limiters", [(1e-6, 1e-6, 1e-6), (1e15, 1e15, 1e15), (1e25, 0.01, 1e25)])
@pytest.mark.parametrize("omega", [0.51, 1.3, 1.9995])
@pytest.mark.parametrize("force", [(0.0, 0.0, 0.0), (1e-3, -2e-3, 5e-4)])
def test_k17_node_at_the_ends(precision, tol, limiters, omega, force):
    O = Oracle(precision)
    p = _lib.FP64 if precision == "f64" else _lib.FP32
    rng = np.random.default_rng(11)
    for _ in range(20):
        f = rng.uniform(-0.5, 0.5, 27) * W
        ref, mref = O.k17_node(f.astype(O.real), omega, limiters, force)
        got, m = lib_node(0, p, f.astype(O.real).astype(np.float64), omega, limiters, force)
        assert np.abs(got - ref).max() / np.abs(ref).max() < tol
        assert np.abs(m - mref).max() / np.abs(mref).max() < tol


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.FP32])
def test_unlimited_by_infinity(precision):
    """An infinite limiter leaves the rate at O: the same as a very large one."""
    f = np.random.default_rng(5).uniform(-0.5, 0.5, 27) * W
    far, _ = lib_node(0, precision, f, 1.8, (1e18,) * 3, (0, 0, 0))
    inf, _ = lib_node(0, precision, f, 1.8, (np.inf,) * 3, (0, 0, 0))
    assert np.all(np.isfinite(inf)) and np.allclose(far, inf, rtol=1e-6 if precision == _lib.FP32 else 1e-14)


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.FP32])
@pytest.mark.parametrize("limiter", [0.0, 1e-35])
def test_limiter_zero_relaxes_fully(precision, limiter):
    """A limiter of zero is the smallest bound (full relaxation), also at rest,
    where the formula as written divides zero by zero."""
    moving = np.random.default_rng(6).uniform(-0.5, 0.5, 27) * W
    for f in (np.zeros(27), moving):
        got, _ = lib_node(0, precision, f, 1.8, (limiter,) * 3, (0, 0, 0))
        full, _ = lib_node(0, precision, f, 1.8, (1e-30,) * 3, (0, 0, 0))
        assert np.all(np.isfinite(got)) and np.allclose(got, full, rtol=0, atol=1e-7 if precision == _lib.FP32 else 1e-15)
