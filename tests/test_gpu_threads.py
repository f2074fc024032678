"""Host threads that use the library at once: launches of one kernel whose shared-memory sizes differ."""

import threading

import numpy as np
import pytest

import stim_gb300
from stim_gb300 import workloads

pytestmark = pytest.mark.gpu


def code(family, distance, p):
    return stim_gb300.Circuit(workloads.code_circuit(family, distance, distance, p))


def in_threads(calls, rounds):
    """Every call `rounds` times in a thread of its own (ctypes releases the interpreter's lock); their results."""
    results, errors = [[] for _ in calls], []
    gate = threading.Barrier(len(calls))

    def work(k):
        try:
            gate.wait()
            for _ in range(rounds):
                results[k].append(calls[k]())
        except Exception as e:  # noqa: BLE001 - shown by the assertion below
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    return results


# Shared memory a CTA takes: 67,584 bytes for d=25, a few KB for d=3; one function serves both.
@pytest.mark.parametrize("mode", [-1, 1])
def test_samplers_of_different_sizes_in_threads(mode):
    circuits = [code("surface_code:rotated_memory_z", d, 1e-3) for d in (3, 25, 3, 25)]
    samplers = [c.compile_detector_sampler(seed=k) for k, c in enumerate(circuits)]
    single = [c.compile_detector_sampler(seed=k) for k, c in enumerate(circuits)]
    for s in samplers:
        s.set_noise_mode(mode)
    rounds = 200 if mode == -1 else 40
    got = in_threads([lambda s=s: s.sample(64, bit_packed=True) for s in samplers], rounds)
    for g, s in zip(got, single):
        for rows in g[:3] + g[-1:]:
            s.set_stream_position(128 * (0 if rows is g[0] else 1 if rows is g[1] else 2 if rows is g[2] else rounds - 1))
            np.testing.assert_array_equal(rows, s.sample(64, bit_packed=True))


def test_converters_of_different_sizes_in_threads():
    circuits = [code("surface_code:rotated_memory_x", d, 5e-3) for d in (3, 15, 3, 15)]
    records = [c.compile_sampler(seed=k).sample(64, bit_packed=True) for k, c in enumerate(circuits)]
    converters = [c.compile_m2d_converter() for c in circuits]
    want = [v.convert(measurements=r, append_observables=True, bit_packed=True) for v, r in zip(converters, records)]
    got = in_threads([lambda v=v, r=r: v.convert(measurements=r, append_observables=True, bit_packed=True)
                      for v, r in zip(converters, records)], 200)
    for g, w in zip(got, want):
        for rows in g:
            np.testing.assert_array_equal(rows, w)
