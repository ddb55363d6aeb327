"""Upload and download with the caller's arrays used in place (page-locked memory, up to 8 MB in all) and copied (any
other): the same bytes arrive, in every order, whatever memory and alignment the arrays have."""
import ctypes as C

import numpy as np
import pytest
import torch

import gfsph

pytestmark = pytest.mark.gpu
CONST = {1: 9.8, 2: 2000.0, 3: 300.0, 5: 5, 9: 0.3, 10: 0.01, 14: 0.5, 15: 0.01}  # 14: the alphas of the pressure at the start


def _array(a, memory, keep):
    """`a` in pageable memory, in page-locked memory, or there four bytes off its alignment."""
    if memory == "pageable":
        return a.copy()
    t = torch.empty(a.nbytes + 64, dtype=torch.uint8).pin_memory()
    keep.append(t)
    off = 4 if memory == "odd" else 0
    out = t.numpy()[off:off + a.nbytes].view(a.dtype).reshape(a.shape)
    out[...] = a
    return out


@pytest.mark.parametrize("flags", [False, True])
@pytest.mark.parametrize("n,memory", [(1, "pinned"), (33, "pinned"), (5003, "pinned"), (5003, "odd"),
                                      (5003, "pageable"), (299_593, "pinned"), (299_594, "pinned")])
def test_same_bytes_in_place_and_copied(gfsph_lib, n, memory, flags):
    rng = np.random.default_rng(n)
    sim = gfsph.Sim(gfsph.make_params(CONST, dt=0.01, icpwp=3, pwp0rel=0.7), np.zeros((64, 64), np.float32), dx=20.0,
                    dy=20.0)
    f4 = np.float32
    a = dict(x=rng.uniform(10, 1200, (n, 2)).astype(f4), v=rng.normal(0, 1, (n, 2)).astype(f4),
             rho=rng.uniform(0.1, 2, n).astype(f4), mass=rng.uniform(1, 2, n).astype(f4),
             hsml=rng.uniform(1, 2, n).astype(f4))
    keep = []
    flag = (rng.random(n) < 0.2).astype(np.int32)
    ins = {k: _array(q, memory, keep) for k, q in a.items()}
    sim.upload(flag=_array(flag, memory, keep) if flags else None, **ins)
    sim.set_time(2.0, 0.25)
    assert sim.step(0)[1] == 2.0
    out = {k: _array(np.full_like(q, 7), memory, keep) for k, q in dict(a, flag=flag).items()}
    sim.download(out=out)
    for k, q in a.items():
        assert np.array_equal(out[k], q), k
    assert np.array_equal(out["flag"], flag if flags else 0 * flag)
    assert np.array_equal(sim.pwp(), f4(0.7) * (a["rho"] * f4(0.5)))
    # only some of the arrays, in other memory than the rest
    v = _array(np.full((n, 2), 7, f4), "pinned", keep)
    h = np.full(n, 7, f4)
    p = lambda q: q.ctypes.data_as(C.POINTER(C.c_float))  # noqa: E731
    assert gfsph.lib().gfsph_download(sim.h, None, p(v), None, None, p(h), None) == 0
    assert np.array_equal(v, a["v"]) and np.array_equal(h, a["hsml"])
    sim.close()
