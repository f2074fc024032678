"""Symptom sampling (symptoms.cu) against the frame kernels and the oracle, bit for bit: every layout it writes, shot
counts around its blocks, destinations at every alignment, windows that move, and gap draws at probabilities where the
float estimate or the gap table decides."""

import numpy as np
import pytest

import stim_gb300
from oracle.oracle import OracleCircuit
from stim_gb300 import _native, workloads
from test_dem_oracle import load_dem
from test_symptoms import HAND

pytestmark = pytest.mark.gpu

CODES = [("surface_code:rotated_memory_z", 3, 0.01), ("surface_code:rotated_memory_z", 5, 0.004),
         ("surface_code:rotated_memory_x", 11, 0.002), ("surface_code:rotated_memory_z", 17, 0.01),
         ("surface_code:rotated_memory_z", 25, 0.001), ("repetition_code:memory", 51, 0.02),
         ("color_code:memory_xyz", 15, 0.005)]


def texts():
    out = {f"{f.split(':')[0]}_d{d}": workloads.code_circuit(f, d, d, p) for f, d, p in CODES}
    out.update(HAND)
    return out


def pair(text, seed):
    """The sampler as it comes, and one that walks the frames."""
    c = stim_gb300.Circuit(text)
    a, b = c.compile_detector_sampler(seed=seed), c.compile_detector_sampler(seed=seed)
    b.set_noise_mode(1)
    return c, a, b


@pytest.mark.parametrize("name", sorted(texts()))
@pytest.mark.parametrize("packed", [True, False])
def test_matches_the_frame_kernels(name, packed):
    c, a, b = pair(texts()[name], 11)
    for shots in (1, 127, 128, 129, 1000):  # the streams go on from call to call
        for kw in ({}, {"append_observables": True}, {"separate_observables": True}, {"prepend_observables": True}):
            x = a.sample(shots, bit_packed=packed, **kw)
            y = b.sample(shots, bit_packed=packed, **kw)
            for u, v in zip(x if isinstance(x, tuple) else (x,), y if isinstance(y, tuple) else (y,)):
                np.testing.assert_array_equal(u, v)


@pytest.mark.parametrize("name", ["surface_code_d3", "surface_code_d17", "surface_code_d25"])
@pytest.mark.parametrize("packed", [True, False])
def test_destinations_at_any_alignment(name, packed):
    torch = pytest.importorskip("torch")
    c, a, b = pair(texts()[name], 5)
    shots = 300
    row = (c.num_detectors + 7) // 8 if packed else c.num_detectors
    want = b.sample(shots, bit_packed=packed).view(np.uint8)
    flags = _native.BIT_PACKED if packed else 0
    for offset, pad in [(k, (5 * k) % 19) for k in range(17)]:
        buf = torch.full((offset + shots * (row + pad) + 64,), 0xA5, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        a.set_stream_position(0)
        _native.check(_native.lib().gfs_sample_detections_device(a._h, shots, flags, buf.data_ptr() + offset, row + pad,
                                                                 None, 0))
        got = buf.cpu().numpy()
        rows = got[offset:offset + shots * (row + pad)].reshape(shots, row + pad)
        np.testing.assert_array_equal(rows[:, :row], want)
        assert (rows[:, row:] == 0xA5).all() and (got[:offset] == 0xA5).all()  # nothing else is written
        assert (got[offset + shots * (row + pad):] == 0xA5).all()


@pytest.mark.parametrize("row", [1, 3, 15, 16, 17, 126, 127, 128])
def test_short_rows_at_any_address(row):
    # Rows around the lengths up to which the kernel writes across rows (16 bytes on the device, 127 in host memory), at
    # addresses of every kind, with nothing written around them.
    torch = pytest.importorskip("torch")
    bits = 8 * row - 3
    qs = " ".join(str(q) for q in range(bits))
    c = stim_gb300.Circuit(f"R {qs}\nX_ERROR(0.2) {qs}\nM {qs}\n" + "".join(f"DETECTOR rec[-{k + 1}]\n" for k in range(bits)))
    a, b = (c.compile_detector_sampler(seed=6) for _ in range(2))
    b.set_noise_mode(1)
    for shots, offset in ((1, 1), (127, 2), (129, 7), (1027, 16), (2000, 3)):
        n = shots * row
        want = b.sample(shots, bit_packed=True)
        dev = torch.full((n + 64,), 0xA5, dtype=torch.uint8, device="cuda")
        host = np.full(n + 64, 0xA5, dtype=np.uint8)
        torch.cuda.synchronize()
        position = a.stream_position()
        _native.check(_native.lib().gfs_sample_detections_device(a._h, shots, _native.BIT_PACKED, dev.data_ptr() + offset, row, None, 0))
        dev = dev.cpu().numpy()
        a.set_stream_position(position)
        a.sample(shots, bit_packed=True, dets_out=host[offset:offset + n].reshape(shots, row))
        for got in (dev, host):
            np.testing.assert_array_equal(got[offset:offset + n].reshape(shots, row), want)
            assert (got[:offset] == 0xA5).all() and (got[offset + n:] == 0xA5).all()


@pytest.mark.parametrize("p", [1e-7, 3e-6, 1e-5, 1e-4, 1e-3, 2.6e-3, 2.8e-3, 0.01, 0.05, 0.2, 0.6, 0.95])
def test_gaps_at_any_probability(p):
    # 40 qubits: two whole segments and a partial one; X flips draw gaps only, depolarizing noise a choice per hit.
    qs = " ".join(str(q) for q in range(40))
    text = (f"R {qs}\nX_ERROR({p}) {qs}\nDEPOLARIZE1({min(p, 0.7)}) {qs}\nM({p}) {qs}\n" +
            "".join(f"DETECTOR rec[-{k + 1}]\n" for k in range(40)) + "OBSERVABLE_INCLUDE(0) rec[-1]\n")
    shots = 1 << 16
    s = stim_gb300.Circuit(text).compile_detector_sampler(seed=3)
    d, o = s.sample(shots, bit_packed=True, separate_observables=True)
    od, oo, _ = OracleCircuit(text).sample(shots, 3)
    np.testing.assert_array_equal(d, od)
    np.testing.assert_array_equal(o, oo)
    assert s.last_timings()["noise_launches"] == 0  # one kernel


def test_a_chosen_frame_kernel_is_used():
    c = stim_gb300.Circuit(texts()["surface_code_d5"])
    want = c.compile_detector_sampler(seed=9).sample(500, bit_packed=True)
    for choose in (lambda s: s.set_noise_mode(1), lambda s: s.set_frame_kernel(1), lambda s: s.set_launch_shape(1, 128)):
        s = c.compile_detector_sampler(seed=9)
        choose(s)
        np.testing.assert_array_equal(s.sample(500, bit_packed=True), want)
        assert s.last_timings()["noise_launches"] == 1


def test_batch_mixes_symptom_and_frame_entries():
    # Small and windowed codes, a circuit whose randomization reaches its outputs, and a sampler with a chosen kernel, in
    # one batch, replayed; then the server with packed and unpacked requests of the same circuits.
    t = texts()
    circuits = [t["surface_code_d3"], t["surface_code_d17"], workloads.random_clifford_circuit(16, 20, 4), t["channels"],
                t["repetition_code_d51"], t["surface_code_d3"]]
    shots = [1000, 300, 129, 1, 4096, 0]
    mk = lambda: [stim_gb300.Circuit(c).compile_detector_sampler(seed=7 + j) for j, c in enumerate(circuits)]
    for kw in ({"bit_packed": True, "separate_observables": True}, {"append_observables": True}):
        ones, many = mk(), mk()
        for s in (ones[4], many[4]):
            s.set_noise_mode(1)
        batch = stim_gb300.BatchSampler(many)
        for _ in range(2):
            for got, s, n in zip(batch.sample(shots, **kw), ones, shots):
                want = s.sample(n, **kw)
                for u, v in zip(got if isinstance(got, tuple) else (got,), want if isinstance(want, tuple) else (want,)):
                    np.testing.assert_array_equal(u, v)
        assert batch.last_timings()["graph_builds"] == 1
    with stim_gb300.Server() as server:
        reqs = [(c, n, packed, server.submit(c, n, seed=50 + j, bit_packed=packed))
                for j, (c, n) in enumerate(zip(circuits, shots)) if n for packed in (True, False)]
        for k, (c, n, packed, r) in enumerate(reqs):
            want = stim_gb300.Circuit(c).compile_detector_sampler(seed=50 + k // 2).sample(n, bit_packed=packed)
            np.testing.assert_array_equal(r.result(), want)


def test_batch_follows_settings_between_calls():
    # Two samplers that trade routes between calls: as many entries each way as before, but not the same ones.
    text = texts()["surface_code_d5"]
    want = [stim_gb300.Circuit(text).compile_detector_sampler(seed=k).sample(900, bit_packed=True) for k in range(2)]
    many = [stim_gb300.Circuit(text).compile_detector_sampler(seed=k) for k in range(2)]
    batch = stim_gb300.BatchSampler(many)
    for modes in ((1, -1), (-1, 1), (-1, -1), (1, 1), (-1, 1)):
        for s, mode in zip(many, modes):
            s.set_stream_position(0)
            s.set_noise_mode(mode)
        for got, w in zip(batch.sample([900, 900], bit_packed=True), want):
            np.testing.assert_array_equal(got, w)


def dem_text(name):
    if name == "surface_rz_d25":
        return workloads.dem_d25_text()
    if name == "hand":  # repeated symptoms, a long list, observables alone, loops, p = 0
        return ("error(0.1) D0 D0 D1\nerror(0.2) L0 L40\nerror(0) D3\nrepeat 9 {\n error(0.01) D0 ^ D1\n"
                " error(0.3) D0 D1 D2 D3 D4 D5 D6 D7 D8 L1\n shift_detectors 3\n}\nerror(0.001) D40\n")
    if name == "far_apart":  # one probability whose mechanisms lie thousands of detectors apart, more than a window
        return "".join(f"error(0.02) D{3000 * k} D{3000 * k + 7} L{k % 3}\nerror(0.0{1 + k % 3}) D{3000 * k + 5}\n"
                       for k in range(20)) + "error(0.02) L2\nerror(0.3) D0\n"
    return str(load_dem(name)["model"])


@pytest.mark.parametrize("name", ["surface_rz_d25", "hand", "far_apart", "rep_d9_r9", "color_d5_r5"])
def test_error_models(name):
    # Without errors returned the model is sampled by its symptoms; with them, mechanism by mechanism.
    text = dem_text(name)
    a, b = (stim_gb300.DetectorErrorModel(text).compile_sampler(seed=21) for _ in range(2))
    for shots in (1, 130, 1000) if name == "surface_rz_d25" else (1, 128, 70001):
        for packed in (True, False):
            d, o, _ = a.sample(shots, bit_packed=packed)
            wd, wo, _ = b.sample(shots, bit_packed=packed, return_errors=True)
            np.testing.assert_array_equal(d, wd)
            np.testing.assert_array_equal(o, wo)


@pytest.mark.parametrize("hits", [0.02, 1.98, 2.02])
@pytest.mark.parametrize("mechanisms", [1, 4, 125, 4 * 16 * 32 + 3, 9001])
def test_error_models_screened(hits, mechanisms):
    # Below two hits a segment (4 mechanisms, 512 trials) a segment's first gap is drawn alone first; around that line, with
    # fewer and more segments than a warp or a CTA has lanes.
    p = hits / 512
    text = "".join(f"error({p!r}) D{k // 2} D{k // 2 + 1}\n" for k in range(mechanisms)) + "logical_observable L0\n"
    a, b = (stim_gb300.DetectorErrorModel(text).compile_sampler(seed=8) for _ in range(2))
    for shots in (1, 129, 20001):
        d, _, _ = a.sample(shots, bit_packed=True)
        wd, _, _ = b.sample(shots, bit_packed=True, return_errors=True)
        np.testing.assert_array_equal(d, wd)


def test_few_and_many_blocks_of_a_large_error_model():
    # The d=25 model (82 K segments a block) changes kernels between 96 and 97 blocks; one stream through either.
    a, b = (stim_gb300.DetectorErrorModel(dem_text("surface_rz_d25")).compile_sampler(seed=3) for _ in range(2))
    for shots in (96 * 128, 96 * 128 + 1):
        d, o, _ = a.sample(shots, bit_packed=True)
        parts = [b.sample(n, bit_packed=True) for n in (50 * 128, shots - 50 * 128)]
        np.testing.assert_array_equal(d, np.concatenate([p[0] for p in parts]))
        np.testing.assert_array_equal(o, np.concatenate([p[1] for p in parts]))


@pytest.mark.parametrize("qubits,shots", [(2, 1), (64, 129), (65, 1000), (128, 513), (130, 300), (300, 140)])
def test_short_phases_around_two_items_a_thread(qubits, shots):
    # The lean frame kernel that works two phases ahead, against the generic one: circuits whose phases have fewer and more
    # items than its threads take (four blocks per CTA: 2 * 256 / 4 = 128 rows), with and without a loop.
    text = workloads.random_clifford_circuit(qubits, 40, 3)
    for t in (text, "REPEAT 3 {\n" + text + "}\n" + text):
        c = stim_gb300.Circuit(t)
        for make in (c.compile_detector_sampler, c.compile_sampler):
            a, b = make(seed=4), make(seed=4)
            b.set_noise_mode(1)
            b.set_frame_kernel(0)
            np.testing.assert_array_equal(a.sample(shots, bit_packed=True), b.sample(shots, bit_packed=True))


@pytest.mark.parametrize("family,distance,ndet_mask", [("surface_code:rotated_memory_z", 3, 2), ("color_code:memory_xyz", 7, 9),
                                                       ("surface_code:rotated_memory_z", 15, 24),
                                                       ("surface_code:rotated_memory_z", 9, 400)])
@pytest.mark.parametrize("shots", [127, 20_011])
def test_decoder_feed_rows_of_any_width(family, distance, ndet_mask, shots):
    # Rows of 3, 21, 421 and 90 bytes, masks of a few bytes and of many, several chunks, against numpy on plain samples.
    text = workloads.code_circuit(family, distance, distance, 0.003)
    c = stim_gb300.Circuit(text)
    bits = np.zeros(c.num_detectors, np.bool_)
    bits[np.random.default_rng(5).choice(c.num_detectors, ndet_mask, replace=False)] = True
    mask = np.packbits(bits, bitorder="little")
    a, b = c.compile_detector_sampler(seed=8), c.compile_detector_sampler(seed=8)
    b.set_noise_mode(1)
    for _ in range(2):
        d, o = b.sample(shots, bit_packed=True, separate_observables=True)
        drop = (d & mask).any(axis=1)
        got = a.sample_for_decoder(shots, postselection_mask=mask)
        np.testing.assert_array_equal(got[0], d[~drop])
        np.testing.assert_array_equal(got[1], o[~drop])
        assert got[2:] == (int(drop.sum()), int(np.unpackbits(d).sum()))
