"""The exact angles of an accepted step (the platform libm's, committed on the
device by the next iteration's first kernel) reach the device within the call
that took the step."""
import numpy as np
import pytest

import sdf_slam_b200 as P
import sdf_slam_b200.scenes as scenes

pytestmark = pytest.mark.gpu


def _room():
    return P.Problem.from_scene(scenes.room_scene(seed=5, grid=40, frames=10, beams=90, max_range=8), P.ProblemOptions())


def test_solve_commits_the_last_steps_angles_before_it_returns():
    """Launches of a solve of i iterations: c + i g + 1, the one being the last
    step's commit (the earlier ones are part of the next iteration)."""
    gpu = _room()
    start = gpu.state()
    launches = []
    for iterations in (0, 1, 2, 3):
        gpu.set_state(*start)
        assert P.solve(gpu, P.SolverOptions(max_iterations=iterations, step_tolerance=0.0)).iterations == iterations
        launches.append(gpu.last_profile()["launches"])
    per_iteration = launches[2] - launches[1]
    assert launches[3] - launches[2] == per_iteration
    assert launches[1] - launches[0] == per_iteration + 1


def test_refused_iteration_keeps_the_angles_of_the_one_before():
    """A launch that fails after an accepted step leaves the state of that step,
    its angles' last bits included (the provisional angles of 299 moved frames
    differ from the libm's in some)."""
    gpu = P.Problem.from_scene(scenes.room_scene(seed=6, grid=40, frames=300, beams=20, max_range=8), P.ProblemOptions())
    start = gpu.state()
    assert P.solve(gpu, P.SolverOptions(max_iterations=1, step_tolerance=0.0)).iterations == 1
    want = gpu.state()
    gpu.set_state(*start)
    gpu.debug_enqueue_fault(1)
    with pytest.raises(RuntimeError, match="refused"):
        P.solve(gpu, P.SolverOptions(max_iterations=3, step_tolerance=0.0))
    got = gpu.state()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    # and the handle goes on from there
    assert P.solve(gpu, P.SolverOptions(max_iterations=2, step_tolerance=0.0)).iterations == 2
