"""Pose Schur complement summed straight into the pose root (pose_schur.cu):
one LM step against the oracle at pose counts around the edges of its 64 x 64
tiles and of the rule that chooses it (256 pose variables), dense and with an
active-region state, and its FP32-front variant against the FP64 step."""
import numpy as np
import pytest

import sdf_slam_b200 as P
import sdf_slam_b200.scenes as scenes
from helpers import oracle_from_specs, rel_err, scene_specs

pytestmark = pytest.mark.gpu

TOL_STEP = 1e-10  # the FP64 path's bound on the step against the oracle


def _warm(frames, active):
    scene = scenes.room_scene(seed=frames, grid=44, frames=frames, beams=40, hallucination_points=2,
                              active_region=active)
    specs, _ = scene_specs(scene)
    orc = oracle_from_specs(specs)
    orc.solve(max_iterations=2, num_threads=4)
    m, p = orc.state()
    return specs, orc, m, p


@pytest.mark.parametrize("frames,active", [(86, False), (87, False), (108, True), (129, False), (150, True)])
def test_pose_schur_step_parity(frames, active):
    # 255 (through the tree), 258, 321, 384 (whole tiles) and 447 pose variables
    specs, orc, m, p = _warm(frames, active)
    gpu = P.Problem.from_specs(specs)
    gpu.set_state(m, p)
    g = gpu.linearize(1.0, False)
    o = orc.linearize(1.0, False, 4, True)
    assert rel_err(g["step"], o["step"]) <= TOL_STEP


def test_pose_schur_mixed_step():
    """FP32 fronts: within an FP32 fraction of the step unrefined, 1e-9 after
    three refinement rounds."""
    specs, _, m, p = _warm(87, False)
    states = []
    for options in [dict(), dict(precision="mixed", refine_steps=0), dict(precision="mixed", refine_steps=3)]:
        gpu = P.Problem.from_specs(specs)
        gpu.set_state(m, p)
        assert P.solve(gpu, P.SolverOptions(max_iterations=1, step_tolerance=0.0, **options)).status == 0
        states.append(np.concatenate([a.ravel() for a in gpu.state()]))
    step = np.max(np.abs(states[0] - np.concatenate([m.ravel(), p.ravel()])))
    assert np.max(np.abs(states[1] - states[0])) <= 1e-3 * step
    assert np.max(np.abs(states[2] - states[0])) <= 1e-9 * step
