"""Scores of a comparison whose kernel gave up waiting (its error word set, as
it does itself): none is left to be taken for a score, and the host is told."""
import glob
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

CPP = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp")


def test_scores_are_invalid(native, tmp_path):
    from sdhash_gb300 import build
    exe = str(tmp_path / "gave_up")
    objs = [o for o in glob.glob(os.path.join(build.BUILD, "*.o")) if not o.endswith("sdbf_compat.o")]
    r = subprocess.run([build._nvcc(), build.ARCH, "-std=c++17", os.path.join(CPP, "gave_up.cc"), *objs, "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
