"""The library's host code against a stand-in for the CUDA runtime (no GPU):
the order of copies and launches over streams, what is read and written where,
and what becomes of errors that no test may cause on a GPU.  The cases are in
tests/cpp/host_paths.cc."""
import glob
import os
import re
import subprocess

import pytest

CPP = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp")
with open(os.path.join(CPP, "host_paths.cc")) as _f:
    CASES = re.findall(r'^    \{"(\w+)", ', _f.read(), flags=re.M)


@pytest.fixture(scope="module")
def program(native, tmp_path_factory):
    from sdhash_gb300 import build
    exe = str(tmp_path_factory.mktemp("host_paths") / "host_paths")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc()))), "include")
    objs = [o for o in glob.glob(os.path.join(build.BUILD, "*.o")) if not o.endswith("sdbf_compat.o")]
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", cuda, os.path.join(CPP, "host_paths.cc"),
                        os.path.join(CPP, "fake_cuda.cc"), *objs, "-o", exe, "-lpthread", "-ldl"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return exe


@pytest.mark.parametrize("case", CASES)
def test_case(program, case):
    r = subprocess.run([program, case], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
