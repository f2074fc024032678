"""The autotuners tune what calls run: the frame kernels' shapes, and sampling by output lists against them."""

import numpy as np
import pytest

import stim_gb300
from stim_gb300 import _native, workloads

pytestmark = pytest.mark.gpu

SHOTS = 1000


def circuit(distance):
    return stim_gb300.Circuit(workloads.code_circuit("surface_code:rotated_memory_z", distance, distance, 1e-3))


def by_lists(s):
    s.sample(SHOTS, bit_packed=True)
    t = s.last_timings()
    return t["noise_launches"] == 0 and t["transpose_launches"] == 0


@pytest.mark.parametrize("trial", [1, 1 << 14])
@pytest.mark.parametrize("distance", [3, 11])
def test_sampler_autotune_keeps_the_fastest(distance, trial):
    # Symptom sampling takes a third of the frame kernels' time or less here, whatever the trial's size; a chosen shape selects
    # the frame kernels until the next measurement.
    s = circuit(distance).compile_detector_sampler(seed=1)
    assert s.autotune(trial) > 0
    assert by_lists(s)
    s.set_launch_shape(1, 64)
    assert not by_lists(s)
    s.autotune(trial)
    assert by_lists(s)


def test_every_setting_can_be_taken_back():
    # Choices that keep detection events on the frame kernels, and what leads back to sampling by output lists.
    s = circuit(5).compile_detector_sampler(seed=1)
    capacity = lambda n: _native.check(_native.lib().gfs_sampler_set_hit_capacity(s._h, n))  # noqa: E731
    for choose, back in ((lambda: s.set_launch_shape(1, 64), lambda: s.set_noise_mode(-1)),
                         (lambda: s.set_noise_mode(1), lambda: s.set_noise_mode(-1)),
                         (lambda: s.set_frame_kernel(0), lambda: s.set_frame_kernel(-1)),
                         (lambda: s.set_ring_placement(1), lambda: s.set_ring_placement(-1)),
                         (lambda: capacity(100), lambda: capacity(0))):
        assert by_lists(s)
        choose()
        assert not by_lists(s)
        back()
    assert by_lists(s)


def test_tuned_frame_kernels_sample_the_same():
    # A chosen noise mode leaves only the frame kernels to tune, and their tuned shape draws the compared bits.
    c = circuit(9)
    a, b = c.compile_detector_sampler(seed=5), c.compile_detector_sampler(seed=5)
    a.set_noise_mode(1)
    assert a.autotune(1 << 14) > 0
    np.testing.assert_array_equal(a.sample(5000, bit_packed=True), b.sample(5000, bit_packed=True))
    assert a.last_timings()["noise_launches"] > 0


@pytest.mark.parametrize("mode", [-1, 1])
def test_batch_autotune_keeps_the_fastest(mode):
    circuits = [circuit(d) for d in (3, 5, 7)]
    samplers = [c.compile_detector_sampler(seed=k) for k, c in enumerate(circuits)]
    single = [c.compile_detector_sampler(seed=k) for k, c in enumerate(circuits)]
    for s in samplers:
        s.set_noise_mode(mode)
    batch = stim_gb300.BatchSampler(samplers)
    shots = [20_000, 3001, 129]
    launches = []

    def check():
        before = batch.last_timings()["transpose_launches"]
        for got, s, n in zip(batch.sample(shots, bit_packed=True), single, shots):
            np.testing.assert_array_equal(got, s.sample(n, bit_packed=True))
        launches.append(batch.last_timings()["transpose_launches"] - before)

    check()
    batch.set_launch_shape(1, 64)
    check()
    assert batch.autotune(shots) > 0
    check()
    assert launches == ([0, 3, 0] if mode == -1 else [3, 3, 3])
