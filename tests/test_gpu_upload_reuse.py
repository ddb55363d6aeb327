"""gfsph_upload has read the caller's arrays when it returns: page-locked ones (read in place up to 8 MB in all, copied
beyond) refilled at once, as a program with one staging buffer for several members does, leave the uploaded state as it
was, also behind work that is still running on the stream."""
import numpy as np
import pytest
import torch

import gfsph

pytestmark = pytest.mark.gpu
CONST = {1: 9.8, 2: 2000.0, 3: 300.0, 5: 5, 9: 0.3, 10: 0.01, 15: 0.01}


@pytest.mark.parametrize("busy", [False, True])
@pytest.mark.parametrize("n", [7, 40_000, 290_000, 400_000])
def test_inputs_refilled_at_once(gfsph_lib, n, busy):
    rng = np.random.default_rng(n)
    f4 = np.float32
    want = dict(x=rng.uniform(10, 1200, (n, 2)).astype(f4), v=rng.normal(0, 1, (n, 2)).astype(f4),
                rho=rng.uniform(0.1, 2, n).astype(f4), mass=rng.uniform(1, 2, n).astype(f4),
                hsml=rng.uniform(1, 2, n).astype(f4), flag=(rng.random(n) < 0.2).astype(np.int32))
    staging = {k: torch.from_numpy(q.copy()).pin_memory().numpy() for k, q in want.items()}
    sim = gfsph.Sim(gfsph.make_params(CONST, dt=0.01), np.zeros((64, 64), f4), dx=20.0, dy=20.0)
    stream = torch.cuda.Stream()
    sim.set_stream(stream.cuda_stream)
    sim.upload(**staging)  # sizes the handle
    if busy:
        with torch.cuda.stream(stream):
            torch.cuda._sleep(20_000_000)  # about 10 ms
    sim.upload(**staging)
    for q in staging.values():
        q[...] = 3
    out = sim.download()
    sim.close()
    for k, q in want.items():
        assert np.array_equal(out[k], q), k
