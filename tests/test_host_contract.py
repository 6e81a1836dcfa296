"""What the entry points ask of the CUDA runtime, checked without a GPU: the
library's host objects linked against the fake runtime of tests/host."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def program(built, tmp_path_factory):
    from rfx_b200 import build

    exe = str(tmp_path_factory.mktemp("host") / "fake_runtime")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.NVCC))), "include")
    subprocess.run([build.HOST_CXX, "-std=c++17", "-O1", "-I" + build.INC, "-I" + build.CSRC, "-I" + cuda, "-o", exe,
                    os.path.join(ROOT, "tests", "host", "fake_runtime.cpp"),
                    os.path.join(build.OBJ, "abi.cu.o"), os.path.join(build.OBJ, "batch.cu.o"),
                    "-Wl,--unresolved-symbols=ignore-all", "-lpthread"], check=True)
    return exe


@pytest.mark.parametrize("scenario", ["other_gpu", "clears", "complete", "tables", "operator_block"])
def test_scenario(program, scenario):
    r = subprocess.run([program, scenario], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
