"""A batch whose launches fail half way is waited for whole (tests/batch_join_check.cc, CUDA stood in for)."""

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
    exe = tmp_path_factory.mktemp("batch_join") / "batch_join_check"
    subprocess.run([cxx, "-std=c++17", "-O1", "-w", "-I", CSRC, "-I", CUDA, os.path.join(HERE, "batch_join_check.cc"),
                    "-Wl,--unresolved-symbols=ignore-all", "-o", str(exe)], check=True)
    return str(exe)


def run(checker, call):
    return subprocess.run([checker, str(call)], capture_output=True, text=True, check=True).stdout


# Calls of four groups: the fork's record and the first launch, three times a wait and a launch, three times a record and a wait.
@pytest.mark.parametrize("call", range(8))
def test_launches_are_waited_for_after_an_error(checker, call):
    launches = [0, 0, 1, 1, 2, 2, 3, 3][call]
    assert run(checker, call) == f"{launches} launches, 0 not waited for, failed\n"


def test_all_launches_are_waited_for(checker):
    assert run(checker, 100) == "4 launches, 0 not waited for, done\n"


@pytest.mark.parametrize("call", range(8, 14))
def test_a_refused_join_leaves_only_its_own_launch(checker, call):
    assert run(checker, call) == "4 launches, 1 not waited for, failed\n"
