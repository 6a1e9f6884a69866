"""Build the sm_100a shared library gems_b200/libgemsgpu.so with nvcc.

The library is built in-tree so that it travels with the repository; the
compile flags pin the B200 target (compute_100a / sm_100a).  The translation
units are compiled side by side into gems_b200/_build and linked.
"""
import concurrent.futures
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "_build")
OUT = os.path.join(HERE, "libgemsgpu.so")
# (object, source, defines): the team kernels once per force-field kind
UNITS = [("gemsgpu", "gemsgpu.cu", []), ("noalloc", "noalloc.cu", []), ("peaks", "peaks.cu", [])] + [
    ("team%d" % k, "team_inst.cu", ["-DTEAM_PART=%d" % k]) for k in range(6)]
DEPS = [os.path.join(CSRC, f) for f in ("gemsgpu.cu", "noalloc.cu", "peaks.cu", "team_inst.cu", "kernels.cuh", "fp64.cuh", "team.cuh",
                                        "lbfgs.cuh", "neb.cuh", "common.cuh")] + [
    os.path.join(os.path.dirname(HERE), "include", "gemsgpu.h")]

NVCC_FLAGS = [
    "-O3", "-std=c++17", "-lineinfo",
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def nvcc():
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if c and os.path.exists(c):
            return c
    raise RuntimeError("nvcc not found")


def stale():
    if not os.path.exists(OUT):
        return True
    t = os.path.getmtime(OUT)
    return any(os.path.getmtime(d) > t for d in DEPS if os.path.exists(d))


def build(force=False, verbose=False, extra=()):
    if not force and not stale():
        return OUT
    os.makedirs(OBJ, exist_ok=True)

    def compile_unit(unit):
        name, src, defines = unit
        obj = os.path.join(OBJ, name + ".o")
        cmd = [nvcc(), *NVCC_FLAGS, *extra, *defines, "-c", "-o", obj, os.path.join(CSRC, src)]
        if verbose:
            print(" ".join(cmd), flush=True)
        subprocess.run(cmd, check=True)
        return obj

    with concurrent.futures.ThreadPoolExecutor(max(1, os.cpu_count() or 1)) as pool:
        objs = list(pool.map(compile_unit, UNITS))
    cmd = [nvcc(), *NVCC_FLAGS, "-shared", "-o", OUT, *objs]
    if verbose:
        print(" ".join(cmd), flush=True)
    subprocess.run(cmd, check=True)
    return OUT


if __name__ == "__main__":
    build(force=True, verbose=True, extra=sys.argv[1:])
