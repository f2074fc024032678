"""Calls in several chunks: a chosen chunk size, page-locked and pageable destinations, the decoder feed's two branches."""

import numpy as np
import pytest

import stim_gb300
from stim_gb300 import workloads

pytestmark = pytest.mark.gpu


def circuit(distance, p=0.01):
    return stim_gb300.Circuit(workloads.code_circuit("surface_code:rotated_memory_z", distance, distance, p))


@pytest.mark.parametrize("mode", [-1, 1])
@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("pinned", [True, False])
def test_a_chosen_chunk_size_is_kept(pinned, packed, mode):
    # 4,100 shots in chunks of 512: nine launches, whatever the size and memory of the result.
    torch = pytest.importorskip("torch")
    c, shots = circuit(5), 4100
    want = c.compile_detector_sampler(seed=2).sample(shots, separate_observables=True, bit_packed=packed)
    s = c.compile_detector_sampler(seed=2)
    s.set_noise_mode(mode)
    s.set_chunk_shots(512)
    dtype = torch.uint8 if packed else torch.bool
    outs = [torch.zeros(w.shape, dtype=dtype, pin_memory=pinned).numpy() for w in want]
    got = s.sample(shots, separate_observables=True, bit_packed=packed, dets_out=outs[0], obs_out=outs[1])
    assert s.last_timings()["frame_launches"] == 9
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)


def test_a_chosen_chunk_size_of_measurements():
    c, shots = circuit(3), 1000
    want = c.compile_sampler(seed=2).sample(shots, bit_packed=True)
    s = c.compile_sampler(seed=2)
    s.set_chunk_shots(512)
    np.testing.assert_array_equal(s.sample(shots, bit_packed=True), want)
    assert s.last_timings()["frame_launches"] == 2


def test_page_locked_rows_of_several_chunks():
    # 110,000 rows of 1,950 bytes: four chunks of 64 MiB, their copies queued as soon as their kernels are.
    torch = pytest.importorskip("torch")
    c, shots = circuit(25, 1e-3), 110_000
    out = torch.zeros((shots, 1950), dtype=torch.uint8, pin_memory=True).numpy()
    s, one = c.compile_detector_sampler(seed=4), c.compile_detector_sampler(seed=4)
    s.sample(shots, bit_packed=True, dets_out=out)
    assert s.last_timings()["frame_launches"] == 4
    for at in range(0, shots, 1 << 15):
        n = min(1 << 15, shots - at)
        np.testing.assert_array_equal(out[at:at + n], one.sample(n, bit_packed=True))


@pytest.mark.parametrize("distance,shots", [(25, 300_000), (3, 20_011)])
def test_decoder_feed_by_frames(distance, shots):
    # A chosen noise mode keeps the feed on the frame kernels: at d=25 in chunks of at most 512 MiB (two here).
    c = circuit(distance, 1e-3)
    bits = np.zeros(c.num_detectors, np.bool_)
    bits[:8] = True
    mask = np.packbits(bits, bitorder="little")
    frames, lists = c.compile_detector_sampler(seed=6), c.compile_detector_sampler(seed=6)
    frames.set_noise_mode(1)
    got = frames.sample_for_decoder(shots, postselection_mask=mask)
    want = lists.sample_for_decoder(shots, postselection_mask=mask)
    assert got[2:] == want[2:]
    for g, w in zip(got[:2], want[:2]):
        np.testing.assert_array_equal(g, w)
