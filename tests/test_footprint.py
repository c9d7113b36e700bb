"""The server's admission estimate against what a handle for the same request
really holds on the device after a solve."""
import re

import pytest

import sdf_slam_b200 as P
import sdf_slam_b200.scenes as scenes
from helpers import scene_specs

pytestmark = pytest.mark.gpu


def _estimate(specs, options):
    """A budget of one byte refuses every request and names its footprint."""
    server = P.Server(1, 1)
    try:
        with pytest.raises(MemoryError) as refused:
            server.submit(specs, options)
    finally:
        server.close()
    return int(re.search(r"footprint (\d+) bytes", str(refused.value)).group(1))


# pose variables below and above the 256 from which the pose Schur complement has
# its own workspace (large beside the fronts on a small grid), wide separators
@pytest.mark.parametrize("grid, frames, beams", [(40, 10, 180), (40, 100, 90), (44, 150, 40), (30, 150, 20),
                                                 (40, 300, 20), (120, 120, 180), (200, 10, 90), (262, 3, 60)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_estimate_covers_what_a_handle_holds(grid, frames, beams, precision):
    specs, _ = scene_specs(scenes.room_scene(seed=3, grid=grid, frames=frames, beams=beams,
                                             max_range=min(30.0, 0.1 * grid + 4)))
    options = P.SolverOptions(max_iterations=2, step_tolerance=0.0, precision=precision)
    estimate = _estimate(specs, options)
    P.release_cached_memory()  # (a cached block may be larger than the one asked for)
    before = P.device_bytes_in_use()
    gpu = P.Problem.from_specs(specs)
    assert P.solve(gpu, options).status == 0
    held = P.device_bytes_in_use() - before
    gpu.close()
    assert P.device_bytes_in_use() == before
    assert held <= estimate <= 2 * held
