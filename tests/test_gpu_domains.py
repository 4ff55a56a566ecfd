"""The persistent fp64 step by domains (vbd_domain.cu): every lanes-per-vertex variant and its
edges -- one domain, partial chunks, vertices with more slots than a lane prefetches, fixed,
free and massless parts -- against the FP64 oracle, and the path for meshes whose domains do
not fit in shared memory against the per-colour graph mode."""
import numpy as np
import pytest

from warpvbd_b200 import BatchedVBDSolver, VBDSolver, _lib, scenes
from oracle.oracle import OracleSolver

pytestmark = pytest.mark.gpu


def _check(kw, steps=3, damping=0.0, material="snh", **opt):
    kw = dict(kw, damping_coefficient=damping, dx_tol=1e-7, max_iter=1000)
    sol = VBDSolver(**kw, mode="persist", material=material, allow_high_valence=True, **opt)
    orc = OracleSolver(**kw, material=material, guarded=True)
    X = kw["initial_positions"]
    diag = float(np.linalg.norm(X.max(0) - X.min(0)))
    for _ in range(steps):
        x = sol.step(sol.old_positions, 1e-3).numpy()
        y = orc.step(None, 1e-3)
        assert sol.last_iterations == orc.last_iterations
        assert np.abs(x - y).max() < 1e-10 * diag
    return sol


@pytest.mark.parametrize("tpv", [0, 2, 4, 8, 16])
@pytest.mark.parametrize("shape,material,damping", [
    ((2, 1, 1), "snh", 0.0),     # 8 solved vertices: one domain
    ((5, 2, 1), "stvk", 0.0),    # 30: two domains
    ((13, 3, 2), "snh", 1.0),    # ragged domains and chunks, the default damping
    ((33, 4, 3), "stvk", 0.0),   # 660: 55 domains
])
def test_domains_match_oracle(shape, material, damping, tpv):
    s = scenes.cantilever(*shape)
    _check(s.solver_kwargs(), material=material, damping=damping, tpv=tpv,
           block_threads=64 if tpv == 2 else 0)


@pytest.mark.parametrize("tpv", [0, 4])
def test_fan_of_many_tets_with_free_and_fixed_vertices(tpv):
    """Two vertices shared by 47 tets (more slots than a lane prefetches), a vertex in no tet
    and fixed vertices."""
    n = 47
    a = np.arange(n + 1) / (n + 1) * 2 * np.pi
    ring = np.stack([np.cos(a), np.sin(a), 0 * a], 1)
    X = np.concatenate([[[0, 0, 0.6], [0, 0, -0.6]], ring, [[3.0, 0, 0]]]) * 0.1
    tets = np.array([[0, 2 + i, 3 + i, 1] for i in range(n)], np.int32)
    active = np.ones(len(X), bool)
    active[2:8] = False
    T = len(tets)
    _check(dict(initial_positions=X, elements=tets, densities=np.full(T, 1000.0),
                youngs_modulus=np.full(T, 5e5), poissons_ratio=np.full(T, 0.4),
                active_mask=active), tpv=tpv)


def test_warm_start_rejected_prediction_is_plain():
    """A network that predicts nonsense is rejected by the potential check: positions and
    sweep counts are the plain step's, bit for bit."""
    from warpvbd_b200 import warmstart
    s = scenes.cantilever(24, 3, 3)
    a = VBDSolver(**s.solver_kwargs(), damping_coefficient=0.0, dx_tol=1e-7, max_iter=1000,
                  mode="persist")
    b = VBDSolver(**s.solver_kwargs(), damping_coefficient=0.0, dx_tol=1e-7, max_iter=1000,
                  mode="persist")
    p = warmstart.init_params(3)
    p[-3:] = 1e4
    b.set_warmstart(p)
    for _ in range(4):
        x = a.step(a.old_positions, 1e-3).numpy()
        y = b.step(b.old_positions, 1e-3).numpy()
        assert a.last_iterations == b.last_iterations
        assert np.array_equal(x, y)


def test_expired_wait_reports_timeout_and_the_solver_recovers():
    s = scenes.cantilever(40)
    p = VBDSolver(**s.solver_kwargs(), damping_coefficient=0.0, dx_tol=1e-7, max_iter=1000,
                  mode="persist")
    L = _lib.load()
    assert L.vbd_set_wait_limits(p._h, 0, 0) == 0
    with pytest.raises(_lib.VBDError) as ei:
        for _ in range(3):
            p.step(p.old_positions, 1e-3)
    assert ei.value.status == _lib.ERR_TIMEOUT
    assert L.vbd_set_wait_limits(p._h, 1 << 26, 2_000_000_000) == 0
    p.reset()
    q = VBDSolver(**s.solver_kwargs(), damping_coefficient=0.0, dx_tol=1e-7, max_iter=1000,
                  mode="persist")
    for _ in range(3):
        assert np.array_equal(p.step(p.old_positions, 1e-3).numpy(),
                              q.step(q.old_positions, 1e-3).numpy())


def test_meshes_whose_domains_do_not_fit_match_graph_mode():
    """320,000 different tets: a domain's records alone exceed a block's shared memory."""
    s = scenes.cantilever(160, 20, 20)
    rng = np.random.default_rng(1)
    s.vertices = s.vertices + rng.uniform(-0.08, 0.08, s.vertices.shape) * s.meta["voxel"]
    kw = dict(s.solver_kwargs(), damping_coefficient=0.0, dx_tol=1e-6, max_iter=1000)
    p, g = VBDSolver(**kw, mode="persist"), VBDSolver(**kw, mode="graph")
    diag = float(np.linalg.norm(s.vertices.max(0) - s.vertices.min(0)))
    for _ in range(2):
        x = p.step(p.old_positions, 1e-3).numpy()
        y = g.step(g.old_positions, 1e-3).numpy()
        assert p.last_iterations == g.last_iterations
        assert np.abs(x - y).max() < 1e-13 * diag


def _steps(solver, n=3):
    out = [np.array(solver.step(1e-3)) for _ in range(n)]
    return out, np.array(solver.positions())


@pytest.mark.parametrize("threads", [64, 128, 256])
def test_environments_that_fill_an_sm_take_the_same_steps_at_any_thread_count(threads):
    """A block whose shared memory leaves no room for another takes 512 threads whatever was
    asked for; small environments beside it and without it take what was asked."""
    large, small = scenes.mass_spring(15, 30), scenes.mass_spring(3, 4)
    for envs in ([large, small], [small, small]):
        runs = []
        for th in (512, threads):
            sol = BatchedVBDSolver(envs, dx_tol=1e-7, max_iter=1000, tiered=True, cluster=2, tpv=4,
                                   block_threads=th)
            runs.append(_steps(sol))
            sol.close()
        assert all((a == b).all() for a, b in zip(runs[0][0], runs[1][0]))
        assert (runs[0][1] == runs[1][1]).all()


def test_environments_set_up_together_are_those_set_up_alone():
    """The setup builds the environments of a batch on several host threads."""
    envs = [scenes.mass_spring(2 + k % 4, 2 + k % 3) for k in range(21)]
    shape = dict(dx_tol=1e-7, max_iter=1000, cluster=1, tpv=4, block_threads=128)
    sol = BatchedVBDSolver(envs, **shape)
    its, x = _steps(sol)
    sol.close()
    at = np.cumsum([0] + [e.n_vertices for e in envs])
    for k, e in enumerate(envs):
        sol = BatchedVBDSolver([e], **shape)
        its1, x1 = _steps(sol)
        sol.close()
        assert [int(i[0]) for i in its1] == [int(i[k]) for i in its]
        assert (x1 == x[at[k]:at[k + 1]]).all()


@pytest.mark.parametrize("polls", [0, 1, 3, 10, 30, 100, 300])
def test_a_step_in_which_a_wait_expired_never_passes_as_finished(polls):
    """With short limits some blocks of a one-sweep step give up, some before the block that
    clears the status has started: the step either reports it or has the whole result."""
    s = scenes.cantilever(40)
    kw = dict(s.solver_kwargs(), damping_coefficient=0.0, dx_tol=1e-7, max_iter=1, mode="persist")
    p, q = VBDSolver(**kw), VBDSolver(**kw)
    ref = q.step(q.old_positions, 1e-3).numpy()
    L = _lib.load()
    assert L.vbd_set_wait_limits(p._h, polls, 2_000_000_000) == 0
    for _ in range(40):
        p.reset()
        try:
            x = p.step(p.old_positions, 1e-3).numpy()
        except _lib.VBDError as e:
            assert e.status == _lib.ERR_TIMEOUT
        else:
            assert np.array_equal(x, ref)
    assert L.vbd_set_wait_limits(p._h, 1 << 26, 2_000_000_000) == 0
    p.reset()
    assert np.array_equal(p.step(p.old_positions, 1e-3).numpy(), ref)


def test_automatic_mode_takes_the_calls_of_block_mode():
    """A mesh that block mode holds, stepped over the whole device by the automatic mode:
    tolerances per environment, the timeline and the direct write of positions."""
    import ctypes
    import torch
    s = scenes.cantilever(40)
    kw = dict(s.solver_kwargs(), damping_coefficient=0.0, dx_tol=1e-7, max_iter=1000)
    a, b = VBDSolver(**kw), VBDSolver(**kw)
    assert a.info()["mode"] == 0x400
    L = _lib.load()
    it = np.zeros(1, np.int32)
    out = torch.empty(s.vertices.shape, dtype=torch.float64).pin_memory().numpy()
    _lib.check(L.vbd_set_trace(a._h, 1))
    for tol in (1e-4, 1e-7):
        x = b.step(b.old_positions, 1e-3, dx_tol=tol).numpy()
        st = L.vbd_step_batched_to(a._h, 1e-3, 1.0, _lib.ptr(np.array([tol]), "d"), 1000,
                                   it.ctypes.data_as(ctypes.POINTER(ctypes.c_int)),
                                   _lib.ptr(out, "d"))
        assert st == _lib.OK
        assert it[0] == b.last_iterations
        assert np.array_equal(out, x)
    n = ctypes.c_int(0)
    _lib.check(L.vbd_get_trace(a._h, None, 0, ctypes.byref(n)))
    rec = np.zeros((n.value, 4), np.uint64)
    _lib.check(L.vbd_get_trace(a._h, rec.ctypes.data_as(ctypes.POINTER(ctypes.c_ulonglong)),
                               n.value, ctypes.byref(n)))
    assert n.value == a.info()["n_blocks"]
    assert (rec[:, 1] > rec[:, 0]).all() and (rec[:, 3] >> np.uint64(8) == it[0]).all()
    # refused before, refused now: the same call in persistent mode by name
    c = VBDSolver(**kw, mode="persist")
    st = L.vbd_step_batched(c._h, 1e-3, 1e-7, _lib.ptr(np.array([1e-7]), "d"), 1000,
                            it.ctypes.data_as(ctypes.POINTER(ctypes.c_int)))
    assert st == _lib.ERR_UNSUPPORTED


def test_automatic_mode_keeps_a_cluster_size_asked_for():
    s = scenes.cantilever(40)
    sol = VBDSolver(**s.solver_kwargs(), damping_coefficient=0.0, cluster=4)
    assert sol.info()["mode"] == 0x100 and sol.info()["cluster"] == 4


@pytest.mark.parametrize("opt", [dict(mode="persist"), dict(mode="block", cluster=1),
                                 dict(mode="block", cluster=4)])
def test_two_lanes_per_vertex_run_as_four(opt):
    s = scenes.cantilever(21, 3, 2)
    kw = dict(s.solver_kwargs(), damping_coefficient=0.0, dx_tol=1e-7, max_iter=1000)
    a, b = (VBDSolver(**kw, **opt, tpv=t, order_index=True) for t in (2, 4))
    for _ in range(3):
        x, y = (v.step(v.old_positions, 1e-3).numpy() for v in (a, b))
        assert a.last_iterations == b.last_iterations and np.array_equal(x, y)


@pytest.mark.parametrize("n", [2, 5, 37])
@pytest.mark.parametrize("warm", [False, True])
def test_plans_that_split_nothing_match_plain_blocks(n, warm):
    """Small equal environments: the plan splits none, whatever the cluster size, and the step
    is that of one block each, the padding of the last cluster included."""
    import torch
    from warpvbd_b200 import warmstart
    envs = [scenes.mass_spring(2 + k % 2, 3) for k in range(n)]
    a = BatchedVBDSolver(envs, dx_tol=1e-7, max_iter=1000)
    b = BatchedVBDSolver(envs, dx_tol=1e-7, max_iter=1000, cluster=1)
    assert a.info()["cluster"] > 1
    if warm:
        a.set_warmstart(warmstart.load())
        b.set_warmstart(warmstart.load())
    out = torch.empty((a.n_vertices, 3), dtype=torch.float64).pin_memory().numpy()
    for _ in range(4):
        assert np.array_equal(a.step(1e-3, out=out), b.step(1e-3))
        assert a.info()["n_blocks"] - n < a.info()["cluster"]
        assert a.info()["block_threads"] == b.info()["block_threads"]
        assert np.array_equal(out, b.positions())


@pytest.mark.parametrize("cube,n,threads", [
    (2, 4, 128),     # a warp or two have chunks
    (5, 4, 256),     # six
    (7, 4, 512),     # sixteen
    (7, 160, 256),   # more environments than SMs: two blocks on one
    (2, 160, 128),
    (15, 160, 512),  # an SM each: its shared memory is full
])
def test_default_thread_count_of_a_batch(cube, n, threads):
    envs = [scenes.mass_spring(cube, 3)] * n
    sol = BatchedVBDSolver(envs, dx_tol=1e-7, max_iter=1000, cluster=1)
    assert sol.info()["block_threads"] == threads
    asked = BatchedVBDSolver(envs[:4], dx_tol=1e-7, max_iter=1000, cluster=1, block_threads=512)
    assert asked.info()["block_threads"] == {2: 128, 5: 256, 7: 512, 15: 512}[cube]
    asked = BatchedVBDSolver(envs[:4], dx_tol=1e-7, max_iter=1000, cluster=1, block_threads=64)
    assert asked.info()["block_threads"] == (512 if cube == 15 else 64)
    its, x = _steps(sol, 2)
    ref = BatchedVBDSolver(envs[:1], dx_tol=1e-7, max_iter=1000, cluster=1, tpv=4,
                           block_threads=64)
    for it in its:
        assert (it == ref.step(1e-3)).all()
    assert (x.reshape(n, -1, 3) == ref.positions()).all()


def test_default_cluster_size_of_a_batch():
    """Six environments take clusters of 16 blocks; eight equal ones with many distinct tets
    take eight blocks each where fewer than eight clusters of 16 fit (seven did)."""
    rng = np.random.default_rng(0)
    heavy = []
    for _ in range(8):
        s = scenes.mass_spring(10, 6)
        s.vertices = s.vertices + rng.uniform(-0.08, 0.08, s.vertices.shape) * s.meta["voxel"]
        heavy.append(s)
    for envs, clusters in ((scenes.env_batch(6, seed=0), (16,)), (heavy, (8, 16))):
        a = BatchedVBDSolver(envs, dx_tol=1e-7, max_iter=1000)
        b = BatchedVBDSolver(envs, dx_tol=1e-7, max_iter=1000, cluster=1)
        assert a.info()["cluster"] in clusters
        for _ in range(3):
            assert np.array_equal(a.step(1e-3), b.step(1e-3))
        assert a.info()["n_blocks"] > len(envs)
        assert np.array_equal(a.positions(), b.positions())


@pytest.mark.parametrize("shape", [(63, 1, 1), (64, 1, 1), (65, 1, 1), (127, 1, 1), (128, 1, 1),
                                   (129, 1, 1), (40, 4, 4)])
def test_domains_set_up_in_groups_are_those_of_one(shape):
    """Host threads take groups of domains from 256 solved vertices on (252, 256, 260; 508,
    512, 516; 1,000): the step is that of one domain, bit for bit at equal lanes."""
    s = scenes.cantilever(*shape)
    kw = dict(s.solver_kwargs(), damping_coefficient=0.0, dx_tol=1e-7, max_iter=1000, tpv=4)
    a, b = VBDSolver(**kw, mode="persist"), VBDSolver(**kw, mode="block", cluster=1)
    assert a.info()["n_blocks"] > 1
    for _ in range(3):
        x, y = (v.step(v.old_positions, 1e-3).numpy() for v in (a, b))
        assert a.last_iterations == b.last_iterations and np.array_equal(x, y)
