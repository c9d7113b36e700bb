"""Accuracy of the factorization and the solve in FP64: products are summed
before they meet the entry they are subtracted from, and systems of large
condition number are solved with a small backward error."""
import numpy as np
import pytest

import sdf_slam_b200 as P
import sdf_slam_b200.scenes as scenes

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("blocks, k", [(1, 63), (1, 64), (2, 64), (5, 64), (20, 64)])
def test_small_products_are_summed_before_they_meet_the_entry(blocks, k):
    """Pivots of one that couple with 2^-27 to a last variable, whose pivot is
    1 - blocks k 2^-54: no product reaches half the last bit of one, so only a
    sum of several does. An 8 x 8 diagonal block may lose its own (seven
    products); the solve adds a few roundings. blocks 1, k 63: one front of 64
    pivots; the others: children of the last variable's front."""
    n = blocks * k + 1
    at = np.arange(n) // k
    pattern = (at[:, None] == at) | (np.arange(n) == n - 1) | (np.arange(n) == n - 1)[:, None]
    a = np.eye(n)
    a[-1, :-1] = a[:-1, -1] = 2.0 ** -27
    cols, rows = np.nonzero(pattern.T)
    solver = P.LdltSolver(n, np.searchsorted(cols, np.arange(n + 1)), rows, np.arange(n))
    solver.factorize(a.T[cols, rows])
    b = np.zeros(n)
    b[-1] = 1.0
    x = solver.solve(b)
    assert abs(x[-1] * (1.0 - blocks * k * 2.0 ** -54) - 1.0) <= 7 * 2.0 ** -54 + 4 * EPS


def _backward_error(apply, row_sum, x, b):
    """|b - A x| / (|A| |x| + |b|), maximum norms, the residual in extended precision."""
    r = b.astype(np.longdouble) - apply(x.astype(np.longdouble))
    return float(np.max(np.abs(r)) / (row_sum * np.max(np.abs(x)) + np.max(np.abs(b))))


@pytest.mark.parametrize("n, shift", [(8, 1e-6), (33, 1e-9), (64, 1e-6), (64, 1e-12), (200, 1e-9)])
def test_chain_with_free_ends(n, shift):
    """Second differences with free ends, shifted: condition number 4 / shift,
    and an inverse of L without small entries. A stable solve's backward error
    is at most 3 n eps."""
    a = 2 * np.eye(n) - np.eye(n, k=1) - np.eye(n, k=-1)
    a[0, 0] = a[-1, -1] = 1.0
    a += shift * np.eye(n)
    outer = np.arange(n + 1) * n
    solver = P.LdltSolver(n, outer, np.tile(np.arange(n), n), np.arange(n))
    solver.factorize(a.ravel())
    rng = np.random.default_rng(n)
    for b in (rng.normal(size=n), np.ones(n), a @ np.sin(np.arange(n) / 7)):
        x = solver.solve(b)
        assert _backward_error(lambda v: a.astype(np.longdouble) @ v, 4.0 + shift, x, b) <= 3 * n * EPS


@pytest.mark.parametrize("grid, frames", [(40, 10), (131, 30), (200, 3)])
@pytest.mark.parametrize("lam", [1.0, 1e-3, 1e-6, 1e-9])
def test_step_at_weak_damping(grid, frames, lam):
    """The step of a damped normal matrix whose condition number grows to 1e12
    and more (separators of up to 200 pivots): backward error at most 64 eps
    (the pivot blocks solve by inverses of up to 256 columns)."""
    scene = scenes.room_scene(seed=grid, grid=grid, frames=frames, beams=90, max_range=0.1 * grid + 4)
    gpu = P.Problem.from_scene(scene, P.ProblemOptions())
    P.solve(gpu, P.SolverOptions(max_iterations=2, step_tolerance=0.0))
    g = gpu.linearize(lam, False)
    begin, rows, values = g["n_outer"][:-1], g["n_inner"], g["n_values"].astype(np.longdouble)
    row_sum = float(np.max(np.add.reduceat(np.abs(g["n_values"]), begin)))
    assert _backward_error(lambda v: np.add.reduceat(values * v[rows], begin), row_sum, g["step"], g["rhs"]) <= 64 * EPS
