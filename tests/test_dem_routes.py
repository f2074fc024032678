"""Which kernels sample an error model's call, on the CPU: the faster ones of the two in measured calls that differ by 15% and
more (tests/dem_route_check.cc)."""

import os
import random
import shutil
import subprocess

import pytest

from stim_gb300 import workloads

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "stim_gb300", "csrc")
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("no C++ compiler or no CUDA headers")
    exe = tmp_path_factory.mktemp("dem_routes") / "dem_route_check"
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC, "-I", CUDA, os.path.join(HERE, "dem_route_check.cc"),
                    os.path.join(CSRC, "dem.cc"), os.path.join(CSRC, "symptoms.cc"), "-o", str(exe)], check=True)
    return str(exe)


def chain(detectors, errors, p, probabilities=2, shuffled=False):
    lines = [f"error({p * (1 + k % probabilities)!r}) " + " ".join(f"D{k * (detectors - 3) // errors + j}" for j in range(3))
             for k in range(errors)]
    if shuffled:
        random.Random(3).shuffle(lines)
    return "\n".join(lines + [f"detector D{detectors - 1}", "logical_observable L0"])


def scattered(detectors, errors, weight):
    rng = random.Random(1)
    return "\n".join([f"error({rng.choice([0.001, 0.002])}) " + " ".join(f"D{d}" for d in rng.sample(range(detectors), weight))
                      for _ in range(errors)] + [f"detector D{detectors - 1}", "logical_observable L0"])


def shuffled_d25():
    lines = workloads.dem_d25_text().splitlines()
    errors = [x for x in lines if x.startswith("error")]
    random.Random(3).shuffle(errors)
    return "\n".join(errors + [x for x in lines if not x.startswith("error")])


# (model, the calls for which symptom sampling measured faster, those for which the mechanism kernels did).
CASES = {
    "d25": (workloads.dem_d25_text, "65536p 131072p", "1p 128p 8192p"),
    "d25 shuffled": (shuffled_d25, "", "1p 129p 65536p"),
    "one window": (lambda: chain(100, 100, 0.001), "1p 1u 129u 65536p 65536u", ""),
    "one window, many hits": (lambda: chain(1000, 5000, 0.3, 1), "1p 1u 4097p 65536u", ""),
    "sparse": (lambda: chain(10000, 400, 0.001), "1p 1u 129p 1025p 16384p", ""),
    "in order": (lambda: chain(10000, 10000, 0.001), "1p 129p 129u 1025p 16384p", ""),
    "many hits": (lambda: chain(10000, 20000, 0.1, 1), "16384p 65536p", "1u 129u 1025u 4097u"),
    "many hits, p=0.3": (lambda: chain(10000, 20000, 0.3, 1), "16384p 65536p", "1p 129p 129u 4097p"),
    "long rows": (lambda: chain(50000, 2000, 0.001), "", "1u 129p 129u 1025p 1025u"),
    "many stages": (lambda: chain(200000, 2000, 0.001), "", "1p 1u 129p 129u 1025p 4097p"),
    "scattered": (lambda: scattered(10000, 20000, 3), "", "129p 2049p"),
    "scattered, long lists": (lambda: scattered(10000, 20000, 30), "", "129p 2049p"),
    "scattered, one window": (lambda: scattered(2000, 20000, 3), "129p 2049p 16384p 65536p", ""),
}


@pytest.mark.parametrize("name", list(CASES))
def test_the_faster_kernels_are_taken(checker, tmp_path, name):
    make, symptoms, mechanisms = CASES[name]
    path = tmp_path / "model.dem"
    path.write_text(make())
    calls = symptoms.split() + mechanisms.split()
    args = [a for c in calls for a in (c[:-1], c[-1])]
    out = subprocess.run([checker, str(path), *args], check=True, capture_output=True, text=True).stdout.split("\n")
    got = dict(zip(calls, out[1:]))
    want = {c: "symptoms" if c in symptoms.split() else "mechanisms" for c in calls}
    assert got == want
