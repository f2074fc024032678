"""Conversions of a few shots: up to 32 turn one group of shots a block, more turn four."""

import numpy as np
import pytest

import stim_gb300
from stim_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("distance", [3, 9, 17])
@pytest.mark.parametrize("shots", [1, 2, 31, 32, 33, 64])
def test_the_first_shots_of_many(distance, shots):
    c = stim_gb300.Circuit(workloads.code_circuit("surface_code:rotated_memory_z", distance, distance, 0.01))
    records = c.compile_sampler(seed=distance).sample(300, bit_packed=True)
    v = c.compile_m2d_converter()
    for kw in ({"append_observables": True}, {"separate_observables": True}):
        many = v.convert(measurements=records, bit_packed=True, **kw)
        few = v.convert(measurements=records[:shots].copy(), bit_packed=True, **kw)
        for m, f in zip(many if isinstance(many, tuple) else (many,), few if isinstance(few, tuple) else (few,)):
            np.testing.assert_array_equal(m[:shots], f)
