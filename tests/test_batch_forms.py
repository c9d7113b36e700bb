"""A small problem's bits do not depend on what shares its handle: alone its cell
pass is one launch and its solve hands values over one by one; beside a member of
more than 512 pose variables the same handle takes one launch per colour and
flags, and merges the levels of all trees."""
import numpy as np
import pytest

import sdf_slam_b200 as P
import sdf_slam_b200.scenes as scenes
from helpers import scene_specs

pytestmark = pytest.mark.gpu


# pose variables: 27, 57 (one front), 177 (tiled, 3 panels); the last member: 537
# (9 panels)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_small_members_beside_a_large_one(precision):
    sizes = [(40, 10), (33, 20), (44, 60), (50, 180)]
    specs = [scene_specs(scenes.room_scene(seed=f, grid=g, frames=f, beams=60, max_range=0.1 * g + 4))[0]
             for g, f in sizes]
    options = P.SolverOptions(max_iterations=4, step_tolerance=0.0, precision=precision)
    batch = P.Problem.batch(specs)
    together = P.solve(batch, options)
    for i, s in enumerate(specs):
        alone = P.Problem.from_specs(s)
        r = P.solve(alone, options)
        assert r.cost_history == together[i].cost_history
        for a, b in zip(alone.state(), batch.state(i)):
            assert np.array_equal(a, b)
