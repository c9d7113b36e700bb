"""Kernel limits (shared memory of the factor and solve kernels) are set on
every device that uses them: the per-device record against a fake of the
attribute call, and two devices of one process where there are two."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import sdf_slam_b200 as P

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_limits_are_raised_on_each_device(tmp_path):
    out = tmp_path / "liblimit_host.so"
    subprocess.run(["g++", "-O1", "-std=c++20", "-shared", "-fPIC", "-I", os.path.join(ROOT, "sdf-slam_b200", "csrc"),
                    os.path.join(ROOT, "tests", "device_limit_host.cpp"), "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))

    def run(start, calls, fail=-1):
        n = len(calls)
        ints = lambda v: (ctypes.c_int * n)(*v)  # noqa: E731
        done = ints([0] * n)
        lib.device_limit_host(start, n, ints([d for d, _ in calls]), ints([v for _, v in calls]), fail, done)
        return list(done)

    # a second device is set though the first one has the value already
    assert run(0, [(0, 100), (0, 100), (1, 100), (1, 100), (0, 100)]) == [1, 0, 1, 0, 0]
    # it only grows, on each device by itself; nothing up to the start value
    assert run(48, [(0, 48), (0, 60), (0, 50), (1, 50), (1, 60), (0, 61)]) == [0, 1, 0, 1, 1, 1]
    # a refused call is made again
    assert run(0, [(3, 10), (3, 10), (3, 10)], fail=0) == [-1, 1, 0]


@pytest.mark.gpu
def test_solves_on_two_devices_of_one_process():
    torch = pytest.importorskip("torch")
    if torch.cuda.device_count() < 2:
        pytest.skip("one device")
    n = 40
    rng = np.random.default_rng(0)
    m = rng.normal(size=(n, n))
    a, b = m @ m.T + n * np.eye(n), rng.normal(size=n)
    x = []
    try:
        for device in (0, 1):
            torch.cuda.set_device(device)
            torch.zeros(1, device="cuda")
            solver = P.LdltSolver(n, np.arange(n + 1) * n, np.tile(np.arange(n), n))
            solver.factorize(a.ravel())
            x.append(solver.solve(b))
            solver.close()
    finally:
        torch.cuda.set_device(0)
    assert np.array_equal(x[0], x[1])
