"""A record conversion that fails half way has read the caller's records and written its arrays for the last time when it
returns (tests/m2d_drain_check.cc, CUDA stood in for)."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "stim_gb300", "csrc")
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("no C++ compiler or no CUDA headers")
    exe = tmp_path_factory.mktemp("m2d_drain") / "m2d_drain_check"
    # Only what the conversion itself calls is stood in for; the rest of the runtime is not linked.
    subprocess.run([cxx, "-std=c++17", "-O1", "-w", "-I", CSRC, "-I", CUDA, os.path.join(HERE, "m2d_drain_check.cc"),
                    "-Wl,--unresolved-symbols=ignore-all", "-o", str(exe)], check=True)
    return str(exe)


# Ten copies out of five chunks, detectors and observables in turn.
@pytest.mark.parametrize("copy", range(11))
def test_nothing_in_flight_after_an_error(checker, copy):
    out = subprocess.run([checker, str(copy)], capture_output=True, text=True, check=True).stdout
    kernels = min(5, copy // 2 + 2)
    assert out == f"{kernels} kernels, 0 in flight, {'failed' if copy < 10 else 'done'}\n"
