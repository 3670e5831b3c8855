"""The adjoint's three schedules of the BC lists: fused (the adjoint's gather and
scatter in one launch, in place), together with separate gathers through a
temporary, and one launch per list.

Tolerances as in tests/test_gpu_adjoint.py: the schedules differ in the order of
the scatters' atomic additions (1e-12); torch autograd through the FP64
transcription 1e-9."""
import numpy as np
import pytest

from tests.test_gpu_adjoint import G, SMALL_BOX, make_sim, problem, torch_reference
from virtualfluids_b200.workloads import adjoint_channel_builder, adjoint_channel_small, inlet_entries, inlet_profile

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SEPARATE = {"fused": None, "together": "VFB_ADJOINT_SEPARATE_GATHERS", "separate": "VFB_ADJOINT_SEPARATE_LISTS"}


@pytest.mark.parametrize("interval", [5, 24])
def test_three_schedules_give_the_same_gradient(cuda, monkeypatch, interval):
    out = []
    for name, variable in SEPARATE.items():
        for v in SEPARATE.values():
            if v:
                monkeypatch.delenv(v, raising=False)
        if variable:
            monkeypatch.setenv(variable, "1")
        sim = make_sim(adjoint_channel_small())
        pb = problem(sim, 24, interval, SMALL_BOX)
        J = pb.evaluate(inlet_profile(sim.levels[0]), G)
        assert sim.adjoint_schedule()["lists_together"] == (name != "separate")
        assert sim.adjoint_fused() == {"lists": name == "fused", "pressure": name == "fused"}
        out.append((J, *pb.gradient(1.0)))
        sim.close()
    J0, dv0, df0 = out[0]
    for J, dv, df in out[1:]:
        assert J == J0
        assert np.abs(dv - dv0).max() <= 1e-12 * np.abs(dv0).max()
        assert np.abs(df - df0).max() <= 1e-12 * np.abs(df0).max()


def test_lists_that_share_cells_are_not_fused(cuda):
    """A cube one node away from the floor, whose floor entries have a link into
    the geometry list's nodes: the first list writes cells that the second reads,
    so each list takes its own launch and gathers first."""
    g = dict(adjoint_channel_builder(16, 8, 8, (6, 2, 2, 8, 4, 4)).arrays()[0])
    k = g["velocity.k"].astype(np.int64)
    up = np.isin(g["neighborY"][k].astype(np.int64), g["geometry.k"]) & ~np.isin(g["neighborY"][k], k)
    assert up.sum() >= 2
    q = g["velocity.q"].reshape(27, -1).copy()
    q[3, up] = 0.5  # the link along +y
    g["velocity.q"] = q.ravel()
    sim = make_sim([g])
    pb = problem(sim, 24, 5, SMALL_BOX)
    profile = inlet_profile(g)
    J = pb.evaluate(profile, G)
    dv, df = sim.adjoint_backward(1.0)
    assert not sim.adjoint_schedule()["lists_together"]
    assert sim.adjoint_fused() == {"lists": False, "pressure": True}
    ref = dict(g)
    ref["velocity.vx"] = g["velocity.vx"].copy()
    ref["velocity.vx"][inlet_entries(g)] = profile
    J_ref, dv_ref, df_ref = torch_reference(ref, 24, profile, G)
    assert abs(J - J_ref) <= 1e-12 * abs(J_ref)
    assert np.abs(dv - dv_ref).max() <= 1e-9 * np.abs(dv_ref).max()
    assert np.abs(df - df_ref).max() <= 1e-9 * np.abs(df_ref).max()
    sim.close()


def test_fused_lists_take_no_gather_scratch(cuda, monkeypatch):
    """27 FP64 values of every BC entry fewer on the device when nothing gathers."""
    taken = []
    for variable in (None, None, "VFB_ADJOINT_SEPARATE_GATHERS"):  # the first run loads the kernels too
        if variable:
            monkeypatch.setenv(variable, "1")
        before = torch.cuda.mem_get_info()[0]
        sim = make_sim(adjoint_channel_builder(128, 64, 64, (40, 26, 26, 52, 38, 38)))
        g = sim.levels[0]
        pb = problem(sim, 4, 2, (80, 96, 24, 40, 24, 40))
        pb.evaluate(inlet_profile(g), G)
        pb.gradient(1.0)
        taken.append(before - torch.cuda.mem_get_info()[0])
        entries = sum(len(g[k]) for k in ("velocity.k", "geometry.k", "pressure0.k"))
        sim.close()
    assert entries > 40000
    assert taken[2] - taken[1] >= 0.75 * 27 * 8 * entries  # the allocator's granularity of 2 MiB a buffer
