"""Single-kernel front factorization (KFactorFront): 8-column panels, row
chunks and shared-memory limits at the edges of their sizes."""
import numpy as np
import pytest

import sdf_slam_b200 as P
import sdf_slam_b200.scenes as scenes
from helpers import oracle_from_specs, rel_err, scene_specs

pytestmark = pytest.mark.gpu


def _csc(a):
    n = len(a)
    outer = np.arange(0, n * n + 1, n)
    inner = np.tile(np.arange(n), n)
    return n, outer, inner, a.T.reshape(-1).copy()


@pytest.mark.parametrize("n", [1, 7, 8, 9, 16, 31, 33, 64, 65, 97, 130, 257])
def test_dense_matrix_solves(n):
    """A dense matrix: supernodes of 64 columns with 0 to n - 64 rows below
    them. Its condition number is below 4, so the solution of LDL^T agrees
    with LU's to a few n eps."""
    rng = np.random.default_rng(n)
    q = rng.normal(size=(n, n))
    a = np.eye(n) + (q + q.T) / (4 * np.sqrt(2 * n))
    n, outer, inner, values = _csc(a)
    solver = P.LdltSolver(n, outer, inner)
    solver.factorize(values)
    b = rng.normal(size=n)
    assert rel_err(solver.solve(b), np.linalg.solve(a, b)) <= 16 * n * np.finfo(float).eps


@pytest.mark.parametrize("at", [0, 7, 9, 40, 63])
def test_zero_pivot_in_any_panel(at):
    a = np.eye(64)
    a[at, at] = 0.0
    n, outer, inner, values = _csc(a)
    solver = P.LdltSolver(n, outer, inner)
    with pytest.raises(RuntimeError):
        solver.factorize(values)
    values[at * 65] = 1.0
    solver.factorize(values)
    assert np.array_equal(solver.solve(np.ones(64)), np.ones(64))


@pytest.mark.parametrize("frames", [2, 4, 33, 34, 43])
def test_pose_root_sizes(frames):
    """Pose roots of 3, 9, 96, 99 and 126 pivots (one kernel up to 128)."""
    scene = scenes.room_scene(seed=frames, grid=41, frames=frames, beams=60, hallucination_points=2)
    specs, _ = scene_specs(scene)
    orc = oracle_from_specs(specs)
    orc.solve(max_iterations=2, num_threads=4)
    m, p = orc.state()
    gpu = P.Problem.from_specs(specs)
    gpu.set_state(m, p)
    g = gpu.linearize(1.0, False)
    o = orc.linearize(1.0, False, 4, True)
    assert rel_err(g["step"], o["step"]) <= 1e-10
