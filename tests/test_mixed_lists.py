"""The lists that only mixed solves read are built when a handle first solves
mixed: a handle that turns mixed, and back, and is analysed again in between,
solves to the bits of handles that were mixed or FP64 from the start."""
import numpy as np
import pytest

import sdf_slam_b200 as P
import sdf_slam_b200.scenes as scenes
from helpers import scene_specs

pytestmark = pytest.mark.gpu


def _solve(gpu, start, precision):
    gpu.set_state(*start)
    r = P.solve(gpu, P.SolverOptions(max_iterations=3, step_tolerance=0.0, precision=precision))
    return [np.array(r.cost_history), *gpu.state()]


# 27 pose variables; 321 (pose columns not stored); wide fronts (tensor cores)
@pytest.mark.parametrize("grid, frames", [(40, 10), (44, 108), (120, 60)])
@pytest.mark.parametrize("between", ["nothing", "schedule", "autotune", "far state"])
def test_handle_that_turns_mixed(grid, frames, between):
    specs, _ = scene_specs(scenes.room_scene(seed=grid, grid=grid, frames=frames, beams=60, max_range=0.1 * grid + 4))
    gpu = P.Problem.from_specs(specs)
    start = gpu.state()
    order = ["fp64", "mixed", "fp64", "mixed"]
    got = []
    for precision in order:
        if between == "schedule":
            gpu.set_schedule(64, 128, 64)
            gpu.set_schedule(128, 256, 128)
        if between == "autotune":
            gpu.autotune()
            gpu.set_schedule(128, 256, 128)
            gpu.set_tensor_core_choice(256)
        if between == "far state":  # every pose elsewhere: a new analysis, then back
            far = start[1].copy()
            far[1:, :2] += 1.0
            gpu.set_state(start[0], far)
            P.solve(gpu, P.SolverOptions(max_iterations=1, step_tolerance=0.0, precision=precision))
        got.append(_solve(gpu, start, precision))
    for precision, g in zip(order, got):
        want = _solve(P.Problem.from_specs(specs), start, precision)
        if between == "far state":  # (a wider pattern sums in another order)
            for a, b in zip(g, want):
                assert np.max(np.abs(a - b)) <= 1e-8 * max(1.0, np.max(np.abs(b)))
        else:
            for a, b in zip(g, want):
                assert np.array_equal(a, b)
