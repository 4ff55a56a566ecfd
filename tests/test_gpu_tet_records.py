"""The fp64 slot path on meshes whose tets are all different, so that the record table takes
each of its three places: staged in shared memory, too large for that (read from global
memory), and past the record count 16-bit slots can name."""
import numpy as np
import pytest

from warpvbd_b200 import VBDSolver, scenes
from oracle.oracle import OracleSolver

pytestmark = pytest.mark.gpu


def _jittered(nx, ny, nz, seed=3):
    s = scenes.cantilever(nx, ny, nz)
    rng = np.random.default_rng(seed)
    s.vertices = s.vertices + rng.uniform(-0.08, 0.08, s.vertices.shape) * s.meta["voxel"]
    return s


@pytest.mark.parametrize("material", ["snh", "stvk"])
@pytest.mark.parametrize("shape,mode,slot_bytes", [
    ((9, 3, 2), "block", 8),     # 270 records: staged
    ((24, 5, 5), "block", 8),    # 3,000 records, 288 KB: read from global memory
    ((24, 5, 5), "persist", 8),  # the same, the whole GPU
    ((24, 5, 5), "graph", 8),
    ((34, 10, 10), "persist", 16),  # 17,000 records: more than 16-bit slots can name
])
def test_distinct_tets_match_oracle(shape, mode, slot_bytes, material):
    s = _jittered(*shape)
    kw = dict(s.solver_kwargs(), damping_coefficient=0.0, dx_tol=1e-7, max_iter=1000)
    sol = VBDSolver(**kw, mode=mode, material=material)
    orc = OracleSolver(**kw, material=material, guarded=True)
    info = sol.info()
    assert info["record_format"] == slot_bytes
    assert info["n_unique_records"] == s.n_tets
    diag = float(np.linalg.norm(s.vertices.max(0) - s.vertices.min(0)))
    for _ in range(3):
        x = sol.step(sol.old_positions, 1e-3).numpy()
        y = orc.step(None, 1e-3)
        assert sol.last_iterations == orc.last_iterations
        # fp64 rounding of two summation orders, as in the other parity tests
        assert np.abs(x - y).max() < 1e-10 * diag
