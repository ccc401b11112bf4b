"""The library's device-memory management (csrc/device_memory.cu) compiled against a CUDA runtime of the host."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("device_memory") / "check")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", cuda, "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "device_memory_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("scenario", ["reuse", "capture", "bound", "give_back", "counts_as_free", "context_in_place",
                                      "context_elsewhere", "no_driver", "host_memory", "threads"])
def test_device_memory(check, scenario):
    r = subprocess.run([check, scenario], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
