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
