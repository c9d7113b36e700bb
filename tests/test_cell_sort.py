"""Cell sort: one and two passes of up to 9 bits, tiles of two and of eight
keys per thread."""
import numpy as np
import pytest

import sdf_slam_b200 as P
import sdf_slam_b200.scenes as scenes
from helpers import oracle_from_specs, rel_err, scene_specs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid, frames, beams, hallucination", [(22, 5, 60, 2), (24, 5, 61, 2), (40, 30, 180, 4),
                                                                (22, 300, 360, 3), (24, 300, 360, 3),
                                                                (60, 300, 360, 3)])
def test_normal_equations_of_sorted_rows(grid, frames, beams, hallucination):
    """The largest three have more rows than fill the GPU with tiles of eight
    keys per thread (303,104), on grids of 441, 529 and 3,481 cells."""
    scene = scenes.room_scene(seed=grid + frames, grid=grid, frames=frames, beams=beams)
    specs, _ = scene_specs(scene, P.ProblemOptions(hallucination_points=hallucination))
    orc = oracle_from_specs(specs)
    gpu = P.Problem.from_specs(specs)
    g = gpu.linearize(1.0, False)
    o = orc.linearize(1.0, False, 4, True)
    assert rel_err(g["step"], o["step"]) <= 1e-10
    again = P.Problem.from_specs(specs).linearize(1.0, False)
    assert np.array_equal(g["step"], again["step"])
