"""Symptom sampling's output lists and stages against a forward walk of the device program, on the CPU
(tests/symptom_check.cc): the same pseudo-random hits at every noise occurrence give the same detectors and observables
through either, for every window size the stages can be planned with."""

import glob
import os
import shutil
import subprocess

import numpy as np
import pytest

from stim_gb300 import workloads

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "stim_gb300", "csrc")

CODES = ["surface_rz_d3_r3", "surface_rz_d25_r25", "surface_rx_d11_r11", "surface_uz_d5_r5", "color_d5_r5",
         "color_d15_r15", "rep_d9_r9", "rep_d51_r51"]

# Loops (one steady from its second-last iteration on, one nested, one whose sets grow), feedback, products, Pauli
# observables, channels of every kind, measurement flips, many observables on one hit, detectors without records.
HAND = {
    "nested": "R 0 1 2\nREPEAT 7 {\n X_ERROR(0.1) 0 1 2\n REPEAT 5 {\n  CX 0 1\n  DEPOLARIZE2(0.05) 0 1 1 2\n  M(0.02) 1\n"
              "  DETECTOR rec[-1]\n }\n MR 2\n DETECTOR rec[-1] rec[-2]\n}\nM 0 1 2\nOBSERVABLE_INCLUDE(3) rec[-1] rec[-2]\n",
    "growing": "R 0 1\nM 1\nREPEAT 60 {\n X_ERROR(0.01) 0\n M 0\n DETECTOR rec[-1]\n}\nM 0\nOBSERVABLE_INCLUDE(0) rec[-1]\n",
    "feedback": "R 0 1 2\nREPEAT 20 {\n PAULI_CHANNEL_1(0.1,0.2,0.05) 0 1\n M(0.1) 0\n CX rec[-1] 1\n CZ rec[-1] 2\n MR 1\n"
                " DETECTOR rec[-1] rec[-2]\n}\n",
    "channels": "R 0 1 2 3\nPAULI_CHANNEL_2(0.01,0.02,0.01,0.02,0.01,0.02,0.01,0.02,0.01,0.02,0.01,0.02,0.01,0.02,0.01) 0 1 2 3\n"
                "Y_ERROR(0.1) 0 1\nZ_ERROR(0.1) 2 3\nM(0.2) 0 1 2 3\nDETECTOR rec[-1] rec[-3]\nDETECTOR\nDETECTOR rec[-2]\n"
                + "".join(f"OBSERVABLE_INCLUDE({k}) rec[-{1 + k % 4}]\n" for k in range(40)),
    "pauli_observable": "RX 0\nR 1\nZ_ERROR(0.2) 0\nX_ERROR(0.3) 1\nOBSERVABLE_INCLUDE(0) X0\nOBSERVABLE_INCLUDE(2) Z1\n",
    "far_apart": "R 0\n" + "R 1\nX_ERROR(0.01) 0\nM 1\nDETECTOR rec[-1]\n" * 400 + "M 0\nDETECTOR rec[-1]\n",
    "quiet_stretch": "R 0 1\nX_ERROR(0.1) 0\nM 0\nDETECTOR rec[-1]\nREPEAT 9000 {\n M 1\n DETECTOR rec[-1]\n}\n"
                     "X_ERROR(0.1) 1\nM 1\nDETECTOR rec[-1]\n",
    # Bodies that give back the state after two and after three iterations, with one and two iterations left over.
    "period_two": "R 0 1\nREPEAT 30 {\n X_ERROR(0.1) 0\n Z_ERROR(0.2) 1\n SWAP 0 1\n H 1\n M(0.1) 0\n}\nR 0 1\n"
                  "REPEAT 21 {\n X_ERROR(0.1) 0 1\n SWAP 0 1\n MR 0\n DETECTOR rec[-1]\n DEPOLARIZE2(0.1) 0 1\n}\n"
                  "M 1\nOBSERVABLE_INCLUDE(1) rec[-1]\n",
    "period_three": "R 0 1 2\nM 0\nREPEAT 40 {\n DEPOLARIZE1(0.1) 0 1 2\n SWAP 0 1 1 2\n MR(0.2) 0\n DETECTOR rec[-1] rec[-2]\n}\n"
                    "M 1 2\nOBSERVABLE_INCLUDE(0) rec[-1] rec[-2]\n",
    "period_five": "R 0 1 2 3 4\nREPEAT 33 {\n DEPOLARIZE1(0.1) 0 1 2 3 4\n SWAP 0 1 1 2 2 3 3 4\n M(0.2) 0\n"
                   " DETECTOR rec[-1]\n}\nM 1 2\nOBSERVABLE_INCLUDE(0) rec[-1] rec[-2]\n",
    "noiseless": "R 0\nM 0\nDETECTOR rec[-1]\n",
}


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path_factory.mktemp("symptoms") / "symptom_check"
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                    os.path.join(HERE, "symptom_check.cc"), os.path.join(CSRC, "lower.cc"),
                    os.path.join(CSRC, "symptoms.cc"), os.path.join(CSRC, "circuit.cc"), "-o", str(exe)], check=True)
    return str(exe)


def run(checker, path):
    out = subprocess.run([checker, path], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    return out.stdout.split()


@pytest.mark.parametrize("name", CODES)
def test_generated_codes(checker, name):
    res = run(checker, os.path.join(workloads.CIRCUIT_DIR, name + ".stim"))
    assert res[0] == "ok"
    stages = [int(x) for x in res[3:]]
    assert stages[0] == 1
    if name == "surface_rz_d25_r25":
        assert max(stages) > 4  # the windowed stages were checked too


@pytest.mark.parametrize("name", sorted(HAND))
def test_hand_circuits(checker, name, tmp_path):
    path = tmp_path / "c.stim"
    path.write_text(HAND[name])
    assert run(checker, str(path))[0] == "ok"


@pytest.mark.parametrize("seed", range(5))
def test_stages_over_random_spans(checker, seed):
    out = subprocess.run([checker, "spans", str(seed)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(HERE, "golden", "*.npz"))), ids=os.path.basename)
def test_reference_fixture_circuits(checker, path, tmp_path):
    g = np.load(path)
    if "circuit" not in g.files:
        pytest.skip("no circuit")
    f = tmp_path / "c.stim"
    f.write_text(str(g["circuit"]))
    assert run(checker, str(f))[0] in ("ok", "no-table")
