"""Error models by either route: symptom sampling and the kernels that go mechanism by mechanism draw the same stream."""

import numpy as np
import pytest

import stim_gb300
from stim_gb300 import workloads

from test_dem_routes import chain, scattered

pytestmark = pytest.mark.gpu

MODELS = {"in order": lambda: chain(10000, 10000, 0.001), "shuffled": lambda: chain(6000, 5003, 0.01, 1, True),
          "many hits": lambda: chain(4001, 2001, 0.3, 1), "scattered": lambda: scattered(9000, 2001, 30),
          "many stages": lambda: chain(50000, 399, 0.01)}


@pytest.mark.parametrize("name", list(MODELS))
def test_every_route(name):
    # With its errors returned the model is sampled mechanism by mechanism; without, by the faster kernels for the call.
    text = MODELS[name]()
    a, b = (stim_gb300.DetectorErrorModel(text).compile_sampler(seed=5) for _ in range(2))
    for shots in (1, 129, 4097, 40001 if name != "many stages" else 12289):
        for packed in (True, False) if shots < 5000 else (True,):
            d, o, _ = a.sample(shots, bit_packed=packed)
            wd, wo, _ = b.sample(shots, bit_packed=packed, return_errors=True)
            np.testing.assert_array_equal(d, wd)
            np.testing.assert_array_equal(o, wo)


@pytest.mark.parametrize("pinned", [False, True])
def test_d25_model_in_several_chunks(pinned):
    # 40,001 shots of 1,951-byte rows: two chunks of 64 MiB by symptom sampling, against calls of 64 blocks, which go
    # mechanism by mechanism.
    torch = pytest.importorskip("torch")
    shots = 40_001
    a, b = (stim_gb300.DetectorErrorModel(workloads.dem_d25_text()).compile_sampler(seed=9) for _ in range(2))
    out = torch.zeros((shots, 1950), dtype=torch.uint8, pin_memory=pinned).numpy()
    d, o, _ = a.sample(shots, bit_packed=True, dets_out=out)
    at = 0
    while at < shots:
        n = min(8192, shots - at)
        wd, wo, _ = b.sample(n, bit_packed=True)
        np.testing.assert_array_equal(d[at:at + n], wd)
        np.testing.assert_array_equal(o[at:at + n], wo)
        at += n
