"""Unpacked rows of symptom sampling: 16-byte units, four of a lane at a time, and the bytes before and after them."""

import numpy as np
import pytest

import stim_gb300
from stim_gb300 import _native

pytestmark = pytest.mark.gpu


def circuit(detectors):
    q = " ".join(map(str, range(detectors)))
    return stim_gb300.Circuit(f"R {q}\nX_ERROR(0.3) {q}\nM {q}\n" + "".join(f"DETECTOR rec[-{k + 1}]\n" for k in range(detectors))
                              + "OBSERVABLE_INCLUDE(0) rec[-1]\n")


# Around one unit, the longest rows written word by word (128), the 32 units of a step, the 128 units of four, and several
# windows (more than 3,072 detectors).
@pytest.mark.parametrize("detectors", [1, 2, 15, 16, 17, 33, 127, 128, 129, 140, 511, 530, 2031, 2048, 2065, 2600, 4000, 9001])
def test_every_alignment(detectors):
    torch = pytest.importorskip("torch")
    c, shots = circuit(detectors), 137
    a, b = c.compile_detector_sampler(seed=3), c.compile_detector_sampler(seed=3)
    b.set_noise_mode(1)
    for append in (False, True):
        want = b.sample(shots, append_observables=append)
        flags = _native.APPEND_OBSERVABLES if append else 0
        at = a.stream_position()
        np.testing.assert_array_equal(a.sample(shots, append_observables=append), want)
        width = want.shape[1]
        for offset, stride in ((0, width + 32 - width % 16), (3, width), (16, width + 1), (7, width + 5)):
            buf = torch.full((offset + stride * shots + 16,), 9, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            a.set_stream_position(at)
            _native.check(_native.lib().gfs_sample_detections_device(a._h, shots, flags, buf.data_ptr() + offset, stride, None, 0))
            got = buf.cpu().numpy()
            rows = np.full((shots, stride), 9, np.uint8)
            rows[:, :width] = want
            np.testing.assert_array_equal(got[offset:offset + stride * shots], rows.reshape(-1))
            assert (got[:offset] == 9).all() and (got[offset + stride * shots:] == 9).all()
