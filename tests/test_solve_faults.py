"""Waits of the one-launch solve that run out: any supernode can be the one that
never publishes, whichever way the solve hands its values over."""
import numpy as np
import pytest

import sdf_slam_b200 as P
import sdf_slam_b200.scenes as scenes

pytestmark = pytest.mark.gpu


# the pose root: one front of 57 pivots; tiled, 3 panels, values handed over
# one by one; tiled, 9 panels, flags
@pytest.mark.parametrize("frames", [20, 60, 180])
@pytest.mark.parametrize("where", ["leaf", "middle", "root"])
def test_withheld_supernode_ends_the_solve(frames, where):
    gpu = P.Problem.from_scene(scenes.room_scene(seed=frames, grid=44, frames=frames, beams=40), P.ProblemOptions())
    P.solve(gpu, P.SolverOptions(max_iterations=1, step_tolerance=0.0))
    count = gpu.debug_supernode_count()
    before = gpu.state()
    gpu.debug_solve_fault({"leaf": 0, "middle": count // 2, "root": count - 1}[where], 4096)
    with pytest.raises(TimeoutError):
        P.solve(gpu, P.SolverOptions(max_iterations=2, step_tolerance=0.0))
    after = gpu.state()
    assert np.array_equal(before[0], after[0]) and np.array_equal(before[1], after[1])
    gpu.debug_solve_fault(-1, 0)
    assert P.solve(gpu, P.SolverOptions(max_iterations=2, step_tolerance=0.0)).iterations == 2


@pytest.mark.parametrize("cell", [0, 20 * 39 + 20, 39 * 39 - 1])
def test_withheld_cell_ends_the_solve(cell):
    """The one-launch cell pass (39 x 39 cells): a corner and a middle cell of the
    first colour, which neighbours wait for; the last corner, of the first colour
    too."""
    gpu = P.Problem.from_scene(scenes.room_scene(seed=4, grid=40, frames=10, beams=90, max_range=8), P.ProblemOptions())
    P.solve(gpu, P.SolverOptions(max_iterations=1, step_tolerance=0.0))
    before = gpu.state()
    gpu.debug_cell_fault(cell, 4096)
    with pytest.raises(TimeoutError):
        P.solve(gpu, P.SolverOptions(max_iterations=2, step_tolerance=0.0))
    after = gpu.state()
    assert np.array_equal(before[0], after[0]) and np.array_equal(before[1], after[1])
    gpu.debug_cell_fault(-1, 0)
    assert P.solve(gpu, P.SolverOptions(max_iterations=2, step_tolerance=0.0)).iterations == 2


def test_fault_hooks_refuse_what_is_out_of_range():
    gpu = P.Problem.from_scene(scenes.room_scene(seed=4, grid=40, frames=10, beams=90, max_range=8), P.ProblemOptions())
    gpu.cost()
    for call in (lambda: gpu.debug_cell_fault(39 * 39), lambda: gpu.debug_cell_fault(-2),
                 lambda: gpu.debug_solve_fault(gpu.debug_supernode_count()), lambda: gpu.debug_solve_fault(-2)):
        with pytest.raises(ValueError):
            call()
