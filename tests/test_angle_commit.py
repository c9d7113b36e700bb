"""The exact angles of an accepted step (the platform libm's, committed on the
device by the next iteration's first kernel) reach the device within the call
that took the step."""
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
