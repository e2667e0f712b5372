"""bench.py's launch count and byte model where y-inverse, z pass and y-forward are
one kernel (8 .. 64 points per side), on the CPU."""
import importlib.util
import os

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("hit3d_bench", os.path.join(REPO, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.mark.parametrize("N", [4, 8, 64, 128])
def test_bytes_of_the_plane_kernel(bench, N):
    b = bench.kernel_alg_bytes(N)
    M, Mz = 2 * (N // 3) + 1, N // 3 + 1
    Bx, Cx = N * M * Mz, N * N * Mz
    plane = 8 <= N <= 64
    assert b["z-pass"] == 9 * (Bx if plane else Cx) * 8
    assert b["y-inverse"] == (0 if plane else 6 * (Bx + Cx) * 8)
    assert b["y-forward"] == (0 if plane else 3 * (Bx + Cx) * 8)


def test_launches_per_step(bench):
    names = ("x-inverse", "y-inverse", "z-pass", "y-forward", "x-forward+epilogue", "forcing-coef")
    assert bench.launches_per_step(dict(zip(names, (1, 8, 8, 8, 8, 8))), 2) == 20
    assert bench.launches_per_step(dict(zip(names, (1, 0, 8, 0, 8, 8))), 2) == 12
