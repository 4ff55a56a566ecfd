"""Meshes that do not run by domains: a vertex that all tets share puts more distinct tets into
one domain (17,000) than its 16-bit slots can name, so the fp64 step runs with persist_kernel
and env_step_kernel, in the shapes measured for those.  Against the FP64 oracle."""
import numpy as np
import pytest

from warpvbd_b200 import BatchedVBDSolver, VBDSolver, scenes
from oracle.oracle import OracleSolver

pytestmark = pytest.mark.gpu


def _hub(n=1500, n_tets=17000, seed=0):
    """A ball: `n` vertices on the sphere, each triangle of near ones joined to the centre."""
    rng = np.random.default_rng(seed)
    i = np.arange(n) + 0.5
    phi, z = np.pi * (1 + 5 ** 0.5) * i, 1 - 2 * i / n
    r = np.sqrt(1 - z * z)
    P = np.stack([r * np.cos(phi), r * np.sin(phi), z], 1) * rng.uniform(0.95, 1.05, (n, 1))
    tri = set()
    for v in range(n):
        near = np.argsort(((P - P[v]) ** 2).sum(1))[1:9]
        for a in range(8):
            for b in range(a + 1, 8):
                t = P[[v, near[a], near[b]]]
                area = np.linalg.norm(np.cross(t[1] - t[0], t[2] - t[0]))
                if area > 0.002:
                    tri.add(tuple(sorted((v, int(near[a]), int(near[b])))))
    tri = np.array(sorted(tri), np.int32)
    assert len(tri) >= n_tets
    tri = tri[np.sort(rng.permutation(len(tri))[:n_tets])]
    X = np.concatenate([P, [[0.0, 0.0, 0.0]]]) * 0.1
    tets = np.concatenate([tri, np.full((len(tri), 1), n, np.int32)], 1).astype(np.int32)
    active = X[:, 2] < 0.08
    T = len(tets)
    return dict(initial_positions=X, elements=tets, densities=np.full(T, 1000.0),
                youngs_modulus=np.full(T, 5e4), poissons_ratio=np.full(T, 0.3),
                active_mask=active)


OPT = dict(damping_coefficient=0.0, dx_tol=1e-7, max_iter=6)


def _oracle(kw, steps, material="snh"):
    orc = OracleSolver(**kw, **OPT, material=material, guarded=True)
    return [(orc.step(None, 1e-3).copy(), orc.last_iterations) for _ in range(steps)]


def _diag(X):
    return float(np.linalg.norm(X.max(0) - X.min(0)))


@pytest.mark.parametrize("material", ["snh", "stvk"])
@pytest.mark.parametrize("opt,kernel,threads", [
    (dict(mode="persist"), "persist_kernel", 128),
    (dict(mode="persist", block_threads=256), "persist_kernel", 256),
    (dict(mode="block", cluster=1), "env_step_kernel", 512),
    (dict(mode="block", cluster=4, block_threads=256), "env_step_kernel", 256),
    (dict(mode="auto"), "env_step_kernel", 512),
])
def test_single_mesh(opt, kernel, threads, material):
    kw = _hub()
    sol = VBDSolver(**kw, **OPT, **opt, material=material, allow_high_valence=True)
    info = sol.info()
    assert info["kernel"] == kernel and info["block_threads"] == threads
    for y, sweeps in _oracle(kw, 2, material):
        x = sol.step(sol.old_positions, 1e-3).numpy()
        assert sol.last_iterations == sweeps
        # fp64 rounding of two summation orders, as in the other parity tests
        assert np.abs(x - y).max() < 1e-10 * _diag(kw["initial_positions"])


@pytest.mark.parametrize("opt", [{}, dict(cluster=1), dict(cluster=2, tiered=True)])
def test_batch_with_such_an_environment(opt):
    small = scenes.mass_spring(4, 5).solver_kwargs()
    envs = [_hub(), small, _hub(seed=1), small]
    sol = BatchedVBDSolver(envs, **OPT, **opt)
    info = sol.info()
    assert info["kernel"] == "env_step_kernel"
    if not opt:
        assert info["cluster"] == 4 and info["block_threads"] == 256
    refs = [_oracle(e, 2) for e in envs]
    for k in range(2):
        it = sol.step(1e-3)
        x = sol.positions()
        for e, ref in enumerate(refs):
            assert it[e] == ref[k][1]
            d = _diag(envs[e]["initial_positions"])
            assert np.abs(x[sol.env_slice(e)] - ref[k][0]).max() < 1e-10 * d


def test_names_of_the_other_kernels():
    s = scenes.cantilever(20)
    kw = dict(s.solver_kwargs(), **OPT)
    for opt, name in ((dict(mode="auto"), "domain_kernel"), (dict(mode="block"), "domain_kernel"),
                      (dict(mode="block", precision="mixed"), "env_step_kernel"),
                      (dict(mode="persist", precision="mixed"), "persist_kernel"),
                      (dict(mode="graph"), "color_kernel")):
        assert VBDSolver(**kw, **opt).info()["kernel"] == name
