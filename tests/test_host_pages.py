"""Pages of the caller's host memory that the device is about to read or write, on the CPU (tests/host_pages_check.cc)."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "stim_gb300", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no C++ compiler or no CUDA headers")
    exe = tmp_path_factory.mktemp("host_pages") / "host_pages_check"
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC, "-I", os.path.join(CUDA, "include"),
                    os.path.join(HERE, "host_pages_check.cc"), "-L", os.path.join(CUDA, "lib64"), "-lcudart_static", "-ldl",
                    "-lrt", "-lpthread", "-o", str(exe)], check=True)
    return str(exe)


def run(checker, case):
    return subprocess.run([checker, case], capture_output=True, text=True)


@pytest.mark.parametrize("case", ["rows_apart", "last_row", "dense"])
def test_only_pages_of_rows_are_asked_for(checker, case):
    out = run(checker, case)
    assert (out.returncode, out.stdout) == (0, "ok\n"), out.stdout + out.stderr


@pytest.mark.parametrize("case", ["read_only", "gaps", "inaccessible"])
def test_memory_that_the_process_may_not_touch_faults_on_the_host(checker, case):
    out = run(checker, case)
    assert (out.returncode, out.stdout) == (0, "ok\n"), out.stdout + out.stderr
