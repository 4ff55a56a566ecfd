"""info() describes what is launched and allocated."""
import pytest

from warpvbd_b200 import BatchedVBDSolver, VBDSolver, autotune, scenes

pytestmark = pytest.mark.gpu
KW = dict(dx_tol=1e-7, max_iter=1000)


def test_lanes_and_threads_as_launched():
    envs = [scenes.mass_spring(4, 3)] * 3
    assert BatchedVBDSolver(envs, **KW, tpv=2).info()["tpv"] == 4
    assert BatchedVBDSolver(envs, **KW, tpv=2, precision="mixed").info()["tpv"] == 2
    s = scenes.cantilever(20)
    sol = VBDSolver(**s.solver_kwargs(), **KW, damping_coefficient=0.0, mode="persist",
                    block_threads=64)
    assert sol.info()["tpv"] == 32 and sol.info()["block_threads"] == 256


def test_device_bytes_count_the_domains():
    """Slots, records and positions of the domains lie beside the solver's: three layouts in a
    batch with a wide tier.  48 bytes a vertex go to the handoff, 8 to every slot."""
    envs = [scenes.mass_spring(6, 5)] * 4
    one = BatchedVBDSolver(envs, **KW, cluster=1).info()
    wide = BatchedVBDSolver(envs, **KW, cluster=4, tiered=True).info()
    graph = VBDSolver(**envs[0].solver_kwargs(), **KW, damping_coefficient=0.0,
                      mode="graph").info()
    n_slots = wide["n_slots"]
    assert one["device_bytes"] > 4 * graph["device_bytes"] + 8 * n_slots
    assert wide["device_bytes"] - one["device_bytes"] > 2 * 8 * n_slots + 48 * wide["n_vertices"]


def test_tuner_reaches_the_automatic_shape(tmp_path):
    """The tuner's space holds the automatic shape, 32 lanes among it, and its result names
    what is launched."""
    kw = scenes.cantilever(40).solver_kwargs()
    cfg = autotune.tune_single(kw, spaces={"persist": autotune.SINGLE_SPACE["persist"]},
                               refresh=True, cache_path=str(tmp_path / "t.json"))
    auto, ran = (VBDSolver(**kw, **KW, damping_coefficient=0.0, **c).info() for c in ({}, cfg))
    assert auto["mode"] == ran["mode"] == 0x400 and auto["tpv"] == 32
    assert cfg["block_threads"] == ran["block_threads"] and cfg["tpv"] in (0, ran["tpv"])


def test_two_lanes_asked_for_take_twice_the_threads():
    kw = dict(scenes.cantilever(20).solver_kwargs(), **KW, damping_coefficient=0.0, mode="block",
              cluster=1)
    for tpv, threads, ran in ((2, 128, 256), (2, 512, 512), (4, 128, 128), (2, 0, 512)):
        info = VBDSolver(**kw, tpv=tpv, block_threads=threads).info()
        assert info["tpv"] == 4 and info["block_threads"] == ran
    mixed = VBDSolver(**kw, precision="mixed", tpv=2, block_threads=128).info()
    assert mixed["tpv"] == 2 and mixed["block_threads"] == 128
