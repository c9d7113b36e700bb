"""One-launch solve (KSolveTree) by pivot block inverses (KInvertFronts): fronts
at the edges of the inverse's tiles and strips, of the row chunks and of the
largest pivot block that is inverted, tiled roots of one and more panels."""
import numpy as np
import pytest

import sdf_slam_b200 as P
import sdf_slam_b200.scenes as scenes
from helpers import oracle_from_specs, rel_err, scene_specs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks, k, border", [(3, 1, 1), (2, 1, 1030), (3, 15, 40), (2, 16, 17), (3, 31, 363),
                                               (2, 33, 341), (3, 48, 1), (2, 63, 178), (5, 64, 175), (2, 64, 176)])
def test_arrow_matrix_solves(blocks, k, border):
    """Dense k x k blocks that couple to a dense border only: fronts of k pivots
    with `border` rows below them (11264 / k - 1 rows make a chunk), whose
    parent has as many children as there are blocks. The condition number is
    below 4, so LDL^T agrees with LU to a few n eps."""
    n = blocks * k + border
    rng = np.random.default_rng(1000 * k + border)
    q = rng.normal(size=(n, n))
    q = (q + q.T) / (4 * np.sqrt(2 * n))
    at = np.minimum(np.arange(n) // k, blocks)
    a = np.eye(n) + np.where((at[:, None] == at) | (at[:, None] == blocks) | (at == blocks), q, 0.0)
    cols, rows = np.nonzero(a.T)
    outer = np.searchsorted(cols, np.arange(n + 1))
    solver = P.LdltSolver(n, outer, rows, np.arange(n))
    solver.factorize(a.T[cols, rows])
    for _ in range(2):
        b = rng.normal(size=n)
        assert rel_err(solver.solve(b), np.linalg.solve(a, b)) <= 16 * n * np.finfo(float).eps


@pytest.mark.parametrize("grid, frames", [(66, 3), (131, 44), (150, 66), (262, 3)])
def test_wide_separators(grid, frames):
    """Top separators past 64 and 128 pivots, and past the largest block that is
    inverted; tiled roots of 129 (three panels) and 195 pivots."""
    scene = scenes.room_scene(seed=grid, grid=grid, frames=frames, beams=60, max_range=0.1 * grid + 4)
    specs, _ = scene_specs(scene)
    orc = oracle_from_specs(specs)
    gpu = P.Problem.from_specs(specs)
    g = gpu.linearize(1.0, False)
    o = orc.linearize(1.0, False, 4, True)
    assert rel_err(g["step"], o["step"]) <= 1e-10
