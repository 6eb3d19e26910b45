"""Host logic that needs no GPU: the library's host-only sources over a fake CUDA runtime (fake_cuda_host.cpp)."""
import os
import subprocess

import pytest

from conftest import PKG, ROOT

SOURCES = ["memory.cu", "host_copy.cu", "host_spmm.cu"]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fake_cuda") / "fake_cuda_host")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.check_call(["g++", "-O1", "-g", "-std=c++17", "-pthread", f"-I{cuda}/include", "-x", "c++", os.path.join(ROOT, "tests", "fake_cuda_host.cpp"),
                           *[os.path.join(PKG, "csrc", f) for f in SOURCES], "-o", exe])
    return exe


@pytest.mark.parametrize("scenario", ["context_device", "pool_under_capture", "staged_copy_fails", "staged_copy_without_threads"])
def test_scenario(program, scenario):
    out = subprocess.run([program, scenario], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
