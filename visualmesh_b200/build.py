"""Builds libvmcuda.so (the CUDA engine and its C ABI) in-tree for sm_100a with nvcc, and the extension module _native (marshalling
for engine.py) against it with g++.

    python -m visualmesh_b200.build            # rebuild what is older than its sources
    python -m visualmesh_b200.build --force [-v]

Every translation unit is compiled to an object file of its own (in parallel) and the objects are linked into the
library; a unit is recompiled when it or one of the headers it includes is newer than its object.
-fmad=false and -ffp-contract=off are part of the contract: the projection arithmetic must round every operation
the way the reference CPU engine does. The graph-convolution kernels call fmaf() explicitly.
"""
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "_build")
LIB = os.path.join(HERE, "libvmcuda.so")
NATIVE = os.path.join(HERE, "_native" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
ABI_HEADER = os.path.join("..", "..", "include", "vmcuda.h")
FFMA_HEADERS = ["conv_ffma_launch.cuh", "conv_ffma.cuh", "conv_common.cuh", "conv_dispatch.hpp", "conv_args.hpp", ABI_HEADER]
# translation unit -> headers it includes (directly or not)
UNITS = {
    "engine.cu": ["kernels.cuh", "tile_plan.cuh", "device_math.cuh", "host_math.hpp", "libm_tables.hpp", "upload.hpp", "conv_dispatch.hpp", "conv_args.hpp",
                  ABI_HEADER],
    "conv_ffma.cu": FFMA_HEADERS,
    "conv_ffma_mid.cu": FFMA_HEADERS,
    "conv_ffma_wide.cu": FFMA_HEADERS,
    "conv_tc.cu": ["conv_tc.cuh", "conv_common.cuh", "conv_dispatch.hpp", "conv_args.hpp", ABI_HEADER],
    "conv_staged.cu": ["conv_staged.cuh", "tile_plan.cuh", "conv_tc.cuh", "conv_common.cuh", "conv_dispatch.hpp", "conv_args.hpp", ABI_HEADER],
    "conv_window.cu": ["conv_window.cuh", "tile_plan.cuh", "conv_tc.cuh", "conv_common.cuh", "conv_dispatch.hpp", "conv_args.hpp", ABI_HEADER],
    "hostmesh.cpp": ["host_math.hpp", ABI_HEADER],
}
NATIVE_SOURCES = ["native.cpp", ABI_HEADER]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    return "nvcc"


def _obj(unit):
    return os.path.join(OBJ, os.path.splitext(unit)[0] + ".o")


def _stale(unit):
    obj = _obj(unit)
    if not os.path.exists(obj):
        return True
    t = os.path.getmtime(obj)
    return any(os.path.getmtime(os.path.join(CSRC, f)) > t for f in [unit] + UNITS[unit]
               if os.path.exists(os.path.join(CSRC, f)))


def needs_build():
    """The library is missing or older than one of its sources (object files may be absent: they do not travel)."""
    return _library_stale() or _native_stale()


def _library_stale():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    files = {f for u in UNITS for f in [u] + UNITS[u]}
    return any(os.path.getmtime(os.path.join(CSRC, f)) > t for f in files if os.path.exists(os.path.join(CSRC, f)))


def _native_stale():
    if not os.path.exists(NATIVE):
        return True
    t = os.path.getmtime(NATIVE)
    return any(os.path.getmtime(os.path.join(CSRC, f)) > t for f in NATIVE_SOURCES if os.path.exists(os.path.join(CSRC, f)))


def build(force=False, verbose=False):
    if force or _library_stale():
        _build_library(force, verbose)
    if force or _native_stale():
        import numpy
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-I", sysconfig.get_paths()["include"],
                        "-I", numpy.get_include(), os.path.join(CSRC, "native.cpp"), "-o", NATIVE, LIB, "-Wl,-rpath,$ORIGIN"],
                       check=True, cwd=CSRC)
    return LIB


def _build_library(force, verbose):
    os.makedirs(OBJ, exist_ok=True)
    flags = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17", "-fmad=false",
             "-Xcompiler", "-fPIC,-ffp-contract=off,-fvisibility=hidden"]
    if verbose:
        flags += ["-Xptxas", "-v"]

    def compile_unit(unit):
        out = subprocess.run([_nvcc()] + flags + ["-c", os.path.join(CSRC, unit), "-o", _obj(unit)], cwd=CSRC,
                             capture_output=True, text=True)
        return unit, out

    todo = [u for u in UNITS if force or _stale(u)]
    with ThreadPoolExecutor(max_workers=max(1, min(len(todo), os.cpu_count() or 1))) as pool:
        for unit, out in pool.map(compile_unit, todo):
            if verbose or out.returncode != 0:
                sys.stderr.write(f"---- {unit}\n{out.stdout}{out.stderr}")
            if out.returncode != 0:
                raise subprocess.CalledProcessError(out.returncode, f"nvcc -c {unit}")
    subprocess.run([_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xlinker", "-soname=libvmcuda.so", "-o", LIB] + [_obj(u) for u in UNITS],
                   check=True, cwd=CSRC)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
