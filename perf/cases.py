"""The work that users of this framework have it do, as cases that can be timed.

A case names a kind of call ("kind"), the circuit or error model it is about, its noise strength, its number of shots and
the options of the call.  ``prepare`` builds what the caller's program holds (a compiled sampler, a converter, a batch, its
output buffers), ``run`` is one call through the public entry points, ``work`` counts the bytes the call has to read and
write.  Every output is bits (packed bytes, or one 0 / 1 byte per bit), so they are compared exactly and no case has a
64-bit reference value (``exact``).

Samplers continue their random stream from call to call, so each pass draws new shots.
"""

import functools
import math
import os

import numpy as np
import torch

import stim_gb300
from stim_gb300 import _native, workloads

SURFACE_Z, SURFACE_X = "surface_code:rotated_memory_z", "surface_code:rotated_memory_x"
REPETITION, COLOR = "repetition_code:memory", "color_code:memory_xyz"

# The distances of each family that have a committed circuit (rounds = distance).
DISTANCES = {SURFACE_Z: range(3, 27, 2), SURFACE_X: range(3, 23, 2), REPETITION: range(3, 53, 2), COLOR: range(3, 17, 2)}

# Committed detector error models: detectors, observables.
MODELS = {"surface_rz_d25_r25": (15600, 1), "surface_rx_d5_r5": (120, 1), "color_d5_r5": (45, 1), "rep_d9_r9": (80, 1)}


def listed():
    return [
        # The smallest call: a thousand shots of a tiny code into numpy, as an interactive user or a test has it.
        {"name": "d3_host_small", "kind": "host", "family": SURFACE_Z, "distance": 3, "p": 1e-3, "shots": 1024,
         "packed": True, "observables": "separate", "pinned": False},
        # The plain arguments (bool arrays, observables appended), an odd number of shots, a noisy repetition code.
        {"name": "rep25_host_bool", "kind": "host", "family": REPETITION, "distance": 25, "p": 1e-2, "shots": 10007,
         "packed": False, "observables": "append", "pinned": False},
        # A threshold study's point: d = 11, p = 5e-3, a million shots left on the device for a decoder there.
        {"name": "d11_device", "kind": "device", "family": SURFACE_X, "distance": 11, "p": 5e-3, "shots": 1 << 20,
         "packed": True},
        # The headline workload: d = 25, 25 rounds, p = 1e-3, 2^20 shots left on the device.
        {"name": "d25_device", "kind": "device", "family": SURFACE_Z, "distance": 25, "p": 1e-3, "shots": 1 << 20,
         "packed": True},
        # The same circuit into the caller's page-locked host arrays, a quarter of the shots.
        {"name": "d25_host_pinned", "kind": "host", "family": SURFACE_Z, "distance": 25, "p": 1e-3, "shots": 1 << 18,
         "packed": True, "observables": "separate", "pinned": True},
        # A medium code at a high error rate and a ragged shot count: many hits per shot.
        {"name": "color13_device_p1e-2", "kind": "device", "family": COLOR, "distance": 13, "p": 1e-2, "shots": 200001,
         "packed": True},
        # Circuits that are no code: random Clifford layers, every measurement a detector, its own p at every layer.
        {"name": "clifford64_device", "kind": "clifford", "qubits": 64, "depth": 200, "circuit_seed": 1,
         "shots": 1 << 17},
        # Measurement records (reference sample XOR flips) of a code, packed, into numpy.
        {"name": "d9_measure", "kind": "measure", "family": SURFACE_Z, "distance": 9, "p": 2e-3, "shots": 65537,
         "packed": True},
        # A sweep over distances and error rates: many circuits of very different sizes in one launch.
        {"name": "batch32_device", "kind": "batch", "circuits": 32, "circuit_seed": 2024, "max_distance": 17,
         "shots_lo": 1 << 10, "shots_hi": 1 << 17},
        # Recorded measurements of an experiment turned into detection events, host arrays in and out.
        {"name": "m2d_d11", "kind": "m2d", "family": SURFACE_X, "distance": 11, "p": 5e-3, "shots": 1 << 18},
        # Sampling a large error model directly.
        {"name": "dem_d25", "kind": "dem", "model": "surface_rz_d25_r25", "shots": 1 << 17, "errors": False},
        # The feed of a decoder: detection events counted, postselected shots dropped, kept rows to the host.
        {"name": "d15_decoder_feed", "kind": "decoder", "family": SURFACE_Z, "distance": 15, "p": 1e-3,
         "shots": 1 << 18, "postselect": 24},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _code(rng, max_distance=25):
    family = rng.choice(sorted(DISTANCES))
    # Repetition codes go twice as far as the others for the same number of qubits and less.
    top = 2 * max_distance + 1 if family == REPETITION else max_distance
    distance = rng.choice([d for d in DISTANCES[family] if d <= top])
    p = float("%.3g" % math.exp(rng.uniform(math.log(1e-4), math.log(1e-2))))
    return {"family": family, "distance": distance, "p": p}


def _cost(family, distance, p):
    """Detectors of the code, weighted up when hits are many: bounds the shots of a drawn case."""
    size = {SURFACE_Z: 1.0, SURFACE_X: 1.0, REPETITION: 2.0 / distance, COLOR: 0.6}[family]
    return size * distance ** 3 * (0.5 + 500 * p)


def _shots(rng, case, lo, hi):
    """Shots spread over [lo, hi], at most as many as the largest listed case's time would allow; odd ones among them."""
    room = _cost(SURFACE_Z, 25, 1e-3) * (1 << 20) / _cost(case["family"], case["distance"], case["p"])
    shots = min(_log_int(rng, lo, hi), int(room))
    return shots | 1 if rng.random() < 0.5 else shots


def draw(rng):
    kind = rng.choice(["host", "host", "device", "device", "device", "clifford", "measure", "batch", "m2d", "dem", "decoder"])
    if kind == "host":
        c = dict(_code(rng), kind=kind, packed=rng.random() < 0.7, observables=rng.choice(["separate", "append", "no"]))
        c["pinned"] = rng.random() < 0.4
        # Up to 2^18 shots of packed rows; unpacked rows are eight times as large.
        c["shots"] = _shots(rng, c, 64, 1 << 18 if c["packed"] else 1 << 15)
        return c
    if kind == "device":
        c = dict(_code(rng), kind=kind, packed=rng.random() < 0.85)
        c["shots"] = _shots(rng, c, 256, 1 << 20 if c["packed"] else 1 << 17)
        return c
    if kind == "clifford":
        n = rng.choice([64, 96, 128, 200, 256])
        return {"kind": kind, "qubits": n, "depth": rng.choice([60, 200]), "circuit_seed": rng.randrange(1, 100),
                "shots": _log_int(rng, 256, (1 << 23) // n)}
    if kind == "measure":
        c = dict(_code(rng, 15), kind=kind, packed=rng.random() < 0.7)
        c["shots"] = _shots(rng, c, 64, 1 << 17 if c["packed"] else 1 << 14)
        return c
    if kind == "batch":
        lo = _log_int(rng, 128, 4096)
        return {"kind": kind, "circuits": rng.randint(4, 40), "circuit_seed": rng.randrange(1, 1000),
                "max_distance": rng.choice([7, 11, 17]), "shots_lo": lo, "shots_hi": lo * rng.choice([4, 32])}
    if kind == "m2d":
        c = dict(_code(rng, 21), kind=kind)
        c["shots"] = _shots(rng, c, 128, 1 << 18)
        return c
    if kind == "dem":
        model = rng.choice(sorted(MODELS))
        big = MODELS[model][0] > 1000
        errors = not big and rng.random() < 0.5
        return {"kind": kind, "model": model, "shots": _log_int(rng, 128, 1 << 16 if big else 1 << 18) | 1,
                "errors": errors}
    c = dict(_code(rng, 21), kind=kind, postselect=rng.choice([0, 8, 40]))
    c["shots"] = _shots(rng, c, 256, 1 << 18)
    return c


@functools.lru_cache(maxsize=None)
def _model_text(name):
    if name == "surface_rz_d25_r25":
        return workloads.dem_d25_text()
    path = os.path.join(os.path.dirname(workloads.CIRCUIT_DIR), "dem", name + ".npz")
    with np.load(path) as z:
        return str(z["model"])


def _text(case):
    return workloads.code_circuit(case["family"], case["distance"], case["distance"], case["p"])


def _batch_list(case):
    distances = tuple(range(3, case["max_distance"] + 2, 2))
    return workloads.batched_workload(case["circuits"], case["circuit_seed"], distances, 1e-4, 1e-2, case["shots_lo"],
                                      case["shots_hi"])


def _host_rows(shots, row, pinned, dtype=torch.uint8):
    """A caller's output array: page-locked, or None for the call to make one."""
    return torch.empty((shots, row), dtype=dtype, pin_memory=True).numpy() if pinned else None


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("host", "device", "decoder"):
        c = stim_gb300.Circuit(_text(case))
        s["sampler"] = c.compile_detector_sampler(seed=seed)
        D, O = c.num_detectors, c.num_observables
    if kind == "host":
        packed = case["packed"]
        nd = D + (O if case["observables"] == "append" else 0)
        if case["pinned"]:
            dtype = torch.uint8 if packed else torch.bool
            s["dets_out"] = _host_rows(case["shots"], (nd + 7) // 8 if packed else nd, True, dtype)
            if case["observables"] == "separate":
                s["obs_out"] = _host_rows(case["shots"], (O + 7) // 8 if packed else O, True, dtype)
    elif kind == "device":
        s["flags"] = _native.BIT_PACKED if case["packed"] else 0
        drow, orow = ((D + 7) // 8, (O + 7) // 8) if case["packed"] else (D, O)
        s["dets"] = torch.empty((case["shots"], drow), dtype=torch.uint8, device="cuda")
        s["obs"] = torch.empty((case["shots"], orow), dtype=torch.uint8, device="cuda")
    elif kind == "clifford":
        text = workloads.random_clifford_circuit(case["qubits"], case["depth"], case["circuit_seed"])
        c = stim_gb300.Circuit(text)
        s["sampler"] = c.compile_detector_sampler(seed=seed)
        s["flags"] = _native.BIT_PACKED
        s["dets"] = torch.empty((case["shots"], (c.num_detectors + 7) // 8), dtype=torch.uint8, device="cuda")
        s["obs"] = None
    elif kind == "measure":
        s["sampler"] = stim_gb300.Circuit(_text(case)).compile_sampler(seed=seed)
    elif kind == "batch":
        s["shots"], samplers, dptr, dstr, optr, ostr, at = [], [], [], [], [], [], 0
        for j, w in enumerate(_batch_list(case)):
            c = stim_gb300.Circuit(w["text"])
            samplers.append(c.compile_detector_sampler(seed=seed * 1000 + j))
            s["shots"].append(w["shots"])
            for ptr, stride, bits in ((dptr, dstr, c.num_detectors), (optr, ostr, c.num_observables)):
                ptr.append(at)
                stride.append((bits + 7) // 8)
                at += -(-w["shots"] * stride[-1] // 16) * 16
        s["arena"] = torch.zeros(at, dtype=torch.uint8, device="cuda")  # every circuit's rows, one after another
        base = s["arena"].data_ptr()
        s["rows"] = ([base + a for a in dptr], dstr, [base + a for a in optr], ostr)
        s["batch"] = stim_gb300.BatchSampler(samplers)
    elif kind == "m2d":
        c = stim_gb300.Circuit(_text(case))
        s["converter"] = c.compile_m2d_converter()
        s["measurements"] = c.compile_sampler(seed=seed).sample(case["shots"], bit_packed=True)
        s["dets_out"] = _host_rows(case["shots"], (c.num_detectors + 7) // 8, True)
        s["obs_out"] = _host_rows(case["shots"], (c.num_observables + 7) // 8, True)
    elif kind == "dem":
        s["sampler"] = stim_gb300.DetectorErrorModel(_model_text(case["model"])).compile_sampler(seed=seed)
        D, O = MODELS[case["model"]]
        s["dets_out"] = _host_rows(case["shots"], (D + 7) // 8, True)
        s["obs_out"] = _host_rows(case["shots"], (O + 7) // 8, True)
    elif kind == "decoder":
        s["mask"] = None
        if case["postselect"]:
            bits = np.zeros(D, dtype=np.bool_)
            bits[:case["postselect"]] = True
            s["mask"] = np.packbits(bits, bitorder="little")
        s["dets_out"] = _host_rows(case["shots"], (D + 7) // 8, True)
        s["obs_out"] = _host_rows(case["shots"], (O + 7) // 8, True)
        s["dets_out"][...] = 0
        s["obs_out"][...] = 0
    if torch.cuda.is_available():
        torch.cuda.synchronize()  # the library works on its own streams: the buffers above exist before it writes them
    return s


def run(s):
    case = s["case"]
    kind, shots = case["kind"], case.get("shots")
    if kind == "host":
        return s["sampler"].sample(shots, bit_packed=case["packed"], append_observables=case["observables"] == "append",
                                   separate_observables=case["observables"] == "separate",
                                   dets_out=s.get("dets_out"), obs_out=s.get("obs_out"))
    if kind in ("device", "clifford"):
        dets, obs = s["dets"], s["obs"]
        _native.check(_native.lib().gfs_sample_detections_device(
            s["sampler"]._h, shots, s["flags"], dets.data_ptr(), dets.shape[1], None if obs is None else obs.data_ptr(),
            0 if obs is None else obs.shape[1]))
        return dets if obs is None else (dets, obs)
    if kind == "measure":
        return s["sampler"].sample(shots, bit_packed=case["packed"])
    if kind == "batch":
        s["batch"].sample_device(s["shots"], *s["rows"])
        return s["arena"]
    if kind == "m2d":
        return s["converter"].convert(measurements=s["measurements"], separate_observables=True, bit_packed=True,
                                      dets_out=s["dets_out"], obs_out=s["obs_out"])
    if kind == "dem":
        return s["sampler"].sample(shots, bit_packed=True, return_errors=case["errors"], dets_out=s["dets_out"],
                                   obs_out=s["obs_out"])
    # The kept rows are the first of the caller's arrays; the arrays are returned whole, so that their shape does not
    # depend on how many shots were kept (the rows after the kept ones are what earlier calls left there).
    kept, _, dropped, events = s["sampler"].sample_for_decoder(shots, postselection_mask=s["mask"],
                                                               dets_out=s["dets_out"], obs_out=s["obs_out"])
    return s["dets_out"], s["obs_out"], len(kept), dropped, events


def work(case):
    kind, shots = case["kind"], case.get("shots")

    def row(bits, packed=True):
        return (bits + 7) // 8 if packed else bits

    if kind == "batch":
        total = 0
        for w in _batch_list(case):
            c = stim_gb300.Circuit(w["text"])
            total += w["shots"] * (row(c.num_detectors) + row(c.num_observables))
        return {"bytes": total, "flops": 0}
    if kind == "dem":
        D, O = MODELS[case["model"]]
        return {"bytes": shots * (row(D) + row(O)), "flops": 0}
    if kind == "clifford":
        c = stim_gb300.Circuit(workloads.random_clifford_circuit(case["qubits"], case["depth"], case["circuit_seed"]))
        return {"bytes": shots * row(c.num_detectors), "flops": 0}
    c = stim_gb300.Circuit(_text(case))
    D, O, M = c.num_detectors, c.num_observables, c.num_measurements
    if kind == "host":
        nd = D + (O if case["observables"] == "append" else 0)
        no = O if case["observables"] == "separate" else 0
        return {"bytes": shots * (row(nd, case["packed"]) + row(no, case["packed"])), "flops": 0}
    if kind == "device":
        return {"bytes": shots * (row(D, case["packed"]) + row(O, case["packed"])), "flops": 0}
    if kind == "measure":
        return {"bytes": shots * row(M, case["packed"]), "flops": 0}
    if kind == "m2d":
        return {"bytes": shots * (row(M) + row(D) + row(O)), "flops": 0}
    return {"bytes": shots * (row(D) + row(O)), "flops": 0}
