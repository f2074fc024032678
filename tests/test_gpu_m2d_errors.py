"""A conversion that fails half way leaves nothing in flight."""

import ctypes

import numpy as np
import pytest

import stim_gb300
from stim_gb300 import _native, workloads

pytestmark = pytest.mark.gpu


def test_records_are_the_callers_again_after_an_error():
    # Six chunks of records that the kernels read where they are.  A device address is no host destination: the first copy out
    # is refused, with kernels of the second chunk queued.  After the error the records may be given away.
    torch = pytest.importorskip("torch")
    c = stim_gb300.Circuit(workloads.code_circuit("surface_code:rotated_memory_x", 11, 11, 5e-3))
    shots, drow = 1 << 18, (c.num_detectors + 7) // 8
    records = c.compile_sampler(seed=1).sample(shots, bit_packed=True)
    converter = c.compile_m2d_converter()
    want = converter.convert(measurements=records, append_observables=False, separate_observables=True, bit_packed=True)
    device = torch.zeros(shots * drow, dtype=torch.uint8, device="cuda")
    lent = records.copy()
    status = _native.lib().gfs_m2d_convert(converter._h, shots, lent.ctypes.data_as(ctypes.c_void_p), lent.strides[0], None, 0,
                                           _native.BIT_PACKED, ctypes.c_void_p(device.data_ptr()), drow, None, 0)
    lent[...] = 0xFF
    del lent
    assert status != 0
    again = converter.convert(measurements=records, append_observables=False, separate_observables=True, bit_packed=True)
    for a, b in zip(again, want):
        np.testing.assert_array_equal(a, b)
