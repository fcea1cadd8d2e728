"""Build the CUDA engine in-tree for sm_100a.

    python -m cudamonsel_b200.build [--force] [-v]

Produces cudamonsel_b200/libcudamonsel_b200.so (C ABI of include/cudamonsel_b200.h).
"""
import argparse
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "libcudamonsel_b200.so")
SOURCES = ["cm_engine.cu"]
DEPS = ["cm_engine.cu", "cm_device.cuh", "cm_physics.cuh", "cm_scene.h", "cm_wave.cuh", "cm_block.cuh", "cm_routes.h", "cm_server.cuh"]
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

# One compilation: -split-compile would take 75 s instead of 200, but inlines otherwise from build to build
# (k_flight_fast spilled 152 to 256 bytes, k_block 20 to 720).
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC",
         "-shared", "-diag-suppress", "20050"]


def stale():
    if not os.path.exists(OUT):
        return True
    t = os.path.getmtime(OUT)
    deps = [os.path.join(CSRC, d) for d in DEPS] + [os.path.join(HERE, "..", "include", "cudamonsel_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    if not force and not stale():
        return OUT
    cmd = [NVCC] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", OUT] + [os.path.join(CSRC, s) for s in SOURCES]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("nvcc failed")
    if verbose:
        sys.stderr.write(r.stderr)
    return OUT


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("-v", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.v))
