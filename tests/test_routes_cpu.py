"""The kernels' short routes (table-search guides, steps strictly inside a region, box tests by reciprocals)
against the general searches, over the forms each accepts: tests/routes/routes.cpp on the CPU."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_routes_agree_with_the_general_searches(tmp_path):
    exe = str(tmp_path / "routes")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-w", "-I", os.path.join(ROOT, "cudamonsel_b200", "csrc"),
                    "-o", exe, os.path.join(HERE, "routes", "routes.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout
