"""Uploads from pageable memory and the libm tables, compiled for the CPU (tests/upload_check.cpp)."""
import os
import subprocess

import pytest

from visualmesh_b200 import build as vm_build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module", params=["this host", "without SSE2"])
def check(tmp_path_factory, request):
    folder = tmp_path_factory.mktemp("upload")
    out, flags = str(folder / "upload_check"), []
    if request.param == "without SSE2":
        # a host that is no x86: the macro is not defined and the header does not exist
        (folder / "emmintrin.h").write_text("#error this host has no SSE2\n")
        flags = ["-U__SSE2__", "-I", str(folder)]
    include = os.path.join(os.path.dirname(os.path.dirname(vm_build._nvcc())), "include")
    subprocess.run(["g++", "-O2", "-std=c++17", *flags, "-I", include, os.path.join(HERE, "upload_check.cpp"), "-o", out, "-lpthread", "-ldl"],
                   check=True)
    return out


# no helper, one of two, all of them
@pytest.mark.parametrize("refused_from", [0, 1, 1000])
def test_every_byte_arrives_however_many_helpers_could_be_started(check, refused_from):
    done = subprocess.run([check, "copies", str(refused_from)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, (done.returncode, done.stdout, done.stderr)


@pytest.mark.parametrize("refused_from", [0, 2])
def test_tables_are_built_with_the_threads_there_are(check, refused_from):
    done = subprocess.run([check, "tables", str(refused_from)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, (done.returncode, done.stdout, done.stderr)
