"""Grid Schur complements pulled by the parents (KChildSchur): more children
than one scan takes, rows at the edges of the 64 x 64 tiles, children of
different depths."""
import numpy as np
import pytest

import sdf_slam_b200 as P
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks, k, border, density", [(15, 3, 64, 1.0), (16, 3, 65, 1.0), (17, 5, 63, 0.5),
                                                        (40, 2, 130, 0.3), (3, 40, 129, 0.5), (2, 64, 257, 0.1)])
def test_blocks_that_share_a_border(blocks, k, border, density):
    """Dense k x k blocks that couple to a random part of a dense border. The
    condition number is below 4, so LDL^T agrees with LU to a few n eps."""
    n = blocks * k + border
    rng = np.random.default_rng(100 * blocks + border)
    q = rng.normal(size=(n, n))
    q = (q + q.T) / (4 * np.sqrt(2 * n))
    at = np.minimum(np.arange(n) // k, blocks)
    keep = (at[:, None] == at) | (at[:, None] == blocks) & (at == blocks)
    couple = rng.uniform(size=(blocks, border)) < density
    for b in range(blocks):
        rows = np.ix_(np.flatnonzero(at == b), blocks * k + np.flatnonzero(couple[b]))
        keep[rows] = True
    keep |= keep.T
    a = np.eye(n) + np.where(keep, q, 0.0)
    cols, rows = np.nonzero(a.T)
    outer = np.searchsorted(cols, np.arange(n + 1))
    solver = P.LdltSolver(n, outer, rows, np.arange(n))
    b = rng.normal(size=n)
    for _ in range(2):
        solver.factorize(a.T[cols, rows])
        assert rel_err(solver.solve(b), np.linalg.solve(a, b)) <= 16 * n * np.finfo(float).eps
