"""Builds ``librivolikernels.so`` (CUDA, sm_100a only) in-tree with nvcc, and ``_launch.so``, Python's calls into it, with g++.

Run as ``python -m rivoli_b200.build``. nvcc cross-compiles without a GPU.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "librivolikernels.so")
LAUNCH = os.path.join(HERE, "_launch.so")
LAUNCH_SRC = os.path.join(CSRC, "python", "launch.cpp")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
    "--fmad=true", "-Xcompiler", "-fPIC,-fvisibility=hidden,-O2", "--shared",
    "-Xptxas", "-v",
]


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "host", "*.cpp")))


def stale() -> bool:
    if not (os.path.exists(OUT) and os.path.exists(LAUNCH)):
        return True
    t = min(os.path.getmtime(OUT), os.path.getmtime(LAUNCH))
    deps = sources() + [LAUNCH_SRC] + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "host", "*.hpp")) + \
        glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def build_launch() -> None:
    """The extension module finds the library beside itself."""
    r = subprocess.run(["/usr/bin/g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-I" + sysconfig.get_path("include"),
                        LAUNCH_SRC, "-o", LAUNCH, "-L" + HERE, "-lrivolikernels", "-Wl,-rpath,$ORIGIN"], capture_output=True, text=True)
    if r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("g++ failed building _launch.so")


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not stale():
        return OUT
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    cmd = [nvcc, *NVCC_FLAGS, "-ccbin", "/usr/bin/g++", "-o", OUT, *sources(), "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
    if r.returncode:
        raise RuntimeError("nvcc failed building librivolikernels.so")
    build_launch()
    # registers / spills / shared memory per kernel: a build log beside the other build products, which are not tracked
    log_dir = os.path.join(HERE, "..", "build")
    os.makedirs(log_dir, exist_ok=True)
    with open(os.path.join(log_dir, "ptxas_info.txt"), "w") as f:
        f.write(r.stdout + r.stderr)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
