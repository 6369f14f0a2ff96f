"""In-tree build of the sm_103a library: nvcc, one translation unit for the C-ABI and
one per neighbour pass and dimension, compiled side by side."""
from __future__ import annotations

import os
import subprocess
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
UNITS = ("armando", "pass_density2d", "pass_density3d", "pass_force2d", "pass_force3d")
OUT = os.path.join(HERE, "lib", "libarmando_gb300.so")

NVCC_FLAGS = [
    "-std=c++17", "-O3", "-lineinfo",
    "-gencode", "arch=compute_103a,code=sm_103a",
    "-Xcompiler", "-fPIC",
    # host code rounds like the oracle on x86 and on Arm (no fused multiply-add)
    "-Xcompiler", "-ffp-contract=off",
]


def sources():
    csrc = os.path.join(HERE, "csrc")
    return [os.path.join(csrc, f) for f in sorted(os.listdir(csrc))
            if f.endswith((".cu", ".cuh", ".h"))] + [
        os.path.join(os.path.dirname(HERE), "include", "armando.h")]


def up_to_date() -> bool:
    if not os.path.exists(OUT):
        return False
    t = os.path.getmtime(OUT)
    return all(os.path.getmtime(s) <= t for s in sources())


def build_library(force: bool = False, verbose: bool = False, extra_flags=()) -> str:
    """Compiles csrc/*.cu into lib/libarmando_gb300.so (skipped when fresh)."""
    if not force and up_to_date():
        return OUT
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    nvcc = os.environ.get("NVCC", "nvcc")

    def run(cmd):
        if verbose:
            print(" ".join(cmd))
        subprocess.run(cmd, check=True)

    with tempfile.TemporaryDirectory(dir=os.path.dirname(OUT)) as tmp:
        objs = [os.path.join(tmp, u + ".o") for u in UNITS]
        cmds = [[nvcc, *NVCC_FLAGS, *extra_flags, "-c", "-o", o, os.path.join(HERE, "csrc", u + ".cu")]
                for u, o in zip(UNITS, objs)]
        with ThreadPoolExecutor(len(cmds)) as ex:
            list(ex.map(run, cmds))
        run([nvcc, *NVCC_FLAGS, "-shared", "-o", OUT, *objs])
    return OUT


if __name__ == "__main__":
    print(build_library(force=True, verbose=True))
