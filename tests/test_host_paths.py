"""Host code of the library without a GPU: its objects linked with tests/cpp/fake_cudart.cpp, a
CUDA runtime on host memory whose calls and launches fail on request, and driven by
tests/cpp/host_paths.cpp.  Covers what no run on a GPU brings about on purpose: error paths,
launch shapes, choices by timing."""
import os
import re
import shutil
import subprocess

import pytest

from conftest import ROOT
from gems_b200 import build

CPP = os.path.join(ROOT, "tests", "cpp")
CASES = re.findall(r"^CASE\((\w+)\)", open(os.path.join(CPP, "host_paths.cpp")).read(), re.M)


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(build.NVCC):
        pytest.skip("no compilers")
    build.build_cuda()
    out = str(tmp_path_factory.mktemp("host_paths") / "host_paths")
    cuda = os.path.dirname(os.path.dirname(build.NVCC))
    subprocess.run(["g++", "-O1", "-std=c++17", "-I" + build.INCLUDE, "-I" + cuda + "/include",
                    os.path.join(CPP, "host_paths.cpp"), os.path.join(CPP, "fake_cudart.cpp")] +
                   [os.path.join(build.BUILD, s + ".o") for s in build.CUDA_SOURCES] +
                   ["-lpthread", "-o", out], check=True)
    return out


@pytest.mark.parametrize("case", CASES)
def test_host_path(exe, case):
    r = subprocess.run([exe, case], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.endswith("OK\n"), r.stdout + r.stderr
