"""The kernels' short routes at the ends of their ranges, on the CPU (tests/routes/edges.cpp)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def edges(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("edges") / "edges")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-w", "-I", os.path.join(ROOT, "cudamonsel_b200", "csrc"),
                    "-o", exe, os.path.join(HERE, "routes", "edges.cpp")], check=True)
    return exe


@pytest.mark.parametrize("what", ["axis_ends", "far_shapes", "fast_models", "grid_walk", "grid_layer"])
def test_short_routes_at_the_ends_of_their_ranges(edges, what):
    r = subprocess.run([edges, what], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout


def test_fast_flights_are_recorded_like_full_ones(tmp_path):
    """tests/routes/trace.cpp: the build that records steps (CM_TRACE)."""
    exe = str(tmp_path / "trace")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-w", "-I", os.path.join(ROOT, "cudamonsel_b200", "csrc"),
                    "-o", exe, os.path.join(HERE, "routes", "trace.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout
