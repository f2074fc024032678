"""Device memory where the host entry points expect host rows: copied to and from, as host memory is, and never touched by the
host."""

import ctypes

import numpy as np
import pytest

import stim_gb300
from stim_gb300 import _native, workloads

pytestmark = pytest.mark.gpu


def device(torch, nbytes):
    b = torch.zeros(max(1, nbytes), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    return b, ctypes.c_void_p(b.data_ptr())


@pytest.mark.parametrize("shots", [100, 5000])
def test_rows_on_the_device(shots):
    torch = pytest.importorskip("torch")
    text = workloads.code_circuit("surface_code:rotated_memory_z", 5, 5, 0.01)
    c = stim_gb300.Circuit(text)
    lib, packed = _native.lib(), _native.BIT_PACKED
    drow, mrow = (c.num_detectors + 7) // 8, (c.num_measurements + 7) // 8
    for mode in (-1, 1):
        want = c.compile_detector_sampler(seed=1).sample(shots, bit_packed=True)
        s = c.compile_detector_sampler(seed=1)
        s.set_noise_mode(mode)
        b, p = device(torch, shots * drow)
        _native.check(lib.gfs_sample_detections(s._h, shots, packed, p, drow, None, 0))
        np.testing.assert_array_equal(b.cpu().numpy().reshape(shots, drow), want)
    records = c.compile_sampler(seed=2, skip_reference_sample=True).sample(shots, bit_packed=True)
    b, p = device(torch, shots * mrow)
    s = c.compile_sampler(seed=2, skip_reference_sample=True)
    _native.check(lib.gfs_sample_measurements(s._h, shots, packed, None, p, mrow))
    np.testing.assert_array_equal(b.cpu().numpy().reshape(shots, mrow), records)
    v = c.compile_m2d_converter()
    want = v.convert(measurements=records, append_observables=False, separate_observables=True, bit_packed=True)[0]
    d, q = device(torch, shots * drow)
    _native.check(lib.gfs_m2d_convert(v._h, shots, p, mrow, None, 0, packed, q, drow, None, 0))
    np.testing.assert_array_equal(d.cpu().numpy().reshape(shots, drow), want)
