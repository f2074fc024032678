"""The one-kernel conversion of bit-packed records (m2d_block.cu) against numpy: record and detector counts around its
32-bit words, short and long lists, expectations, both observable layouts, shots around its 128-shot blocks, and a circuit
too large for it, through the general path."""

import numpy as np
import pytest

import stim_gb300

pytestmark = pytest.mark.gpu


def circuit(M, lists, obs):
    """M measurements of X-flipped qubits (reference 1 for odd ones), detectors and observables over absolute records."""
    t = "".join(f"X {k}\n" for k in range(1, M, 2)) + "M " + " ".join(str(k) for k in range(M)) + "\n"
    t += "".join("DETECTOR " + " ".join(f"rec[-{M - i}]" for i in d) + "\n" for d in lists)
    return t + "".join(f"OBSERVABLE_INCLUDE({k}) " + " ".join(f"rec[-{M - i}]" for i in o) + "\n" for k, o in enumerate(obs))


@pytest.mark.parametrize("M,D,O", [(1, 1, 0), (7, 0, 3), (31, 33, 1), (32, 32, 33), (33, 95, 0), (129, 64, 40), (1441, 1320, 1),
                                   (3000, 700, 2), (5000, 4000, 1)])
@pytest.mark.parametrize("shots", [1, 127, 300, 9000])
def test_against_numpy(M, D, O, shots):
    rng = np.random.default_rng(M * 1000 + D)
    pick = lambda k: sorted(rng.choice(M, size=min(M, k), replace=False).tolist())
    lists = [pick(int(rng.integers(0, 10))) for _ in range(D)]  # none to nine: eight is the short lists' limit
    obs = [pick(int(rng.integers(1, 60))) for _ in range(O)]
    c = stim_gb300.Circuit(circuit(M, lists, obs))
    m = rng.integers(0, 2, size=(shots, M), dtype=np.uint8).astype(np.bool_)
    ref = np.arange(M) % 2 == 1
    fold = lambda ls: np.array([(m[:, l].sum(axis=1) + ref[l].sum()) % 2 for l in ls], np.bool_).reshape(len(ls), shots).T
    wd, wo = fold(lists), fold(obs)
    packed = np.packbits(m, axis=1, bitorder="little")
    conv = c.compile_m2d_converter()
    pack = lambda a: np.packbits(a, axis=1, bitorder="little")
    d, o = conv.convert(measurements=packed, separate_observables=True, bit_packed=True)
    np.testing.assert_array_equal(d, pack(wd))
    np.testing.assert_array_equal(o, pack(wo))
    both = conv.convert(measurements=packed, append_observables=True, bit_packed=True)
    np.testing.assert_array_equal(both, pack(np.concatenate([wd, wo], axis=1)))
    np.testing.assert_array_equal(conv.convert(measurements=m, append_observables=True),
                                  np.concatenate([wd, wo], axis=1))
