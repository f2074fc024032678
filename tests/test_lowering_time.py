"""Lowering takes time in proportion to the circuit: the backward pass that finds the output lists must not cost many times
what the rest does."""

import time

import stim_gb300


def seconds(text, tries=3):
    c = stim_gb300.Circuit(text)
    best = 1e9
    for _ in range(tries):
        t0 = time.perf_counter()
        c.program_info()
        best = min(best, time.perf_counter() - t0)
    return best


def test_many_short_loops_over_many_qubits():
    # Each loop iteration touches one of 5,000 qubits; copying the state of all of them for every loop took 100 times as long.
    q = " ".join(map(str, range(5000)))
    end = f"M {q}\n" + "".join(f"DETECTOR rec[-{k + 1}]\n" for k in range(5000))
    body = "H 0\nX_ERROR(0.01) 0\n"
    looped = seconds(f"R {q}\n" + ("REPEAT 2 {\n" + body + "}\n") * 1000 + end)
    flat = seconds(f"R {q}\n" + (body + body) * 1000 + end)
    assert looped < 10 * flat + 0.05


def test_lists_too_long_to_pay():
    # No resets, every result a detector: a hit flips all later results of its qubit.  Listing them took ten times as long as
    # lowering, and the sampler then kept its frames.
    q = " ".join(map(str, range(200)))

    def raw(noise):
        return (f"R {q}\nREPEAT 200 {{\n{noise}M {q}\n" + "".join(f"DETECTOR rec[-{k + 1}]\n" for k in range(200)) + "}\n")

    assert seconds(raw(f"DEPOLARIZE1(0.01) {q}\n")) < 4 * seconds(raw("")) + 0.02
