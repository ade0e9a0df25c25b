"""Copies into host memory (host_copy.hpp) over a stand-in for the CUDA runtime,
no GPU: page-locked destinations, no page-locked memory for the slots, no
memory at all."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("host_copy") / "host_copy"
    cpp = os.path.join(ROOT, "tests", "cpp")
    r = subprocess.run([os.environ.get("NICP_CXX", "g++"), "-std=c++17", "-O1", "-pthread",
                        "-I", os.path.join(cpp, "fake_cuda"), "-I", os.path.join(ROOT, "nicp_b200", "csrc"),
                        os.path.join(cpp, "host_copy.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return str(exe)


@pytest.mark.parametrize("scenario", ["locked", "no_slots", "no_memory"])
def test_host_copier(program, scenario):
    r = subprocess.run([program, scenario], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
