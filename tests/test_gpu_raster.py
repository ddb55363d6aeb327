"""The depth raster and the hazard statistics against their definitions, particle by particle, for particles in any
order: in runs of one DEM cell and alone, on and beyond the edges of the DEM, and with a depth that is not finite."""
import ctypes as C

import numpy as np
import pytest
import torch

import gfsph

pytestmark = pytest.mark.gpu
f4 = np.float32


def _particles(n, nx, ny, cell, order, seed):
    rng = np.random.default_rng(seed)
    lo, hi = (-3 * cell, (nx + 3) * cell) if order == "beyond" else (0.0, (nx - 1) * cell)
    x = rng.uniform(lo, hi, (n, 2)).astype(f4)
    x[:, 1] *= f4((ny + 2.0) / (nx + 2.0))
    if order == "runs":
        x = x[np.lexsort((x[:, 0] // cell, x[:, 1] // cell))]
    x[:: 97] = np.round(x[:: 97] / cell) * f4(cell)  # on the nodes
    h = rng.uniform(0.1, 5.0, n).astype(f4)
    if n > 200:
        h[n // 2] = np.inf
    return x, rng.normal(0, 3, (n, 2)).astype(f4), h


def _idw(x, h, nx, ny, cell):
    """Sums of h/d and 1/d with 32-bit terms and 64-bit sums."""
    acc = np.zeros((2, ny, nx))
    c = f4(cell)
    distg = np.sqrt(c * c + c * c)
    ipx, ipy = (x[:, 0] / c + f4(1)).astype(np.int64), (x[:, 1] / c + f4(1)).astype(np.int64)
    for ox in range(-1, 3):
        for oy in range(-1, 3):
            ix, iy = ipx + ox, ipy + oy
            ok = (ix >= 1) & (ix <= nx) & (iy >= 1) & (iy <= ny)
            ddx, ddy = x[ok, 0] - (ix[ok] - 1).astype(f4) * c, x[ok, 1] - (iy[ok] - 1).astype(f4) * c
            d = np.maximum(np.sqrt(ddx * ddx + ddy * ddy), f4(1e-6)) / distg
            for a, t in ((acc[0], h[ok] / d), (acc[1], f4(1) / d)):
                np.add.at(a, (iy[ok] - 1, ix[ok] - 1), t.astype(np.float64))
    return acc


@pytest.mark.parametrize("n,nx,ny,order", [(1, 8, 8, "runs"), (33, 4, 5, "runs"), (5003, 33, 21, "runs"),
                                           (5003, 64, 64, "alone"), (4001, 16, 40, "beyond")])
def test_raster_and_hazard_against_their_sums(gfsph_lib, n, nx, ny, order):
    cell = 2.0
    x, v, h = _particles(n, nx, ny, cell, order, n + nx)
    sim = gfsph.Sim(gfsph.make_params({1: 9.8, 2: 2000.0, 3: 300.0, 5: 5, 9: 0.3, 10: 0.01, 15: 0.01}, dt=0.01,
                                      h_inf=0.0), np.zeros((ny, nx), f4), dx=cell, dy=cell)
    sim.upload(x, v, h, np.ones(n, f4), np.ones(n, f4))
    acc = _idw(x, h, nx, ny, cell)
    with np.errstate(invalid="ignore", divide="ignore"):
        want = np.where(acc[1].astype(f4) >= f4(1e-6), acc[0] / acc[1], acc[0]).astype(f4)
    # the same terms, summed in 64 bits in another order: at most the last place of the 32-bit result differs
    np.testing.assert_allclose(sim.raster(gfsph.RASTER_DEPTH_IDW), want, rtol=2.0 ** -23)

    ix = np.clip((x[:, 0] / f4(cell) + f4(1)).astype(np.int64), 1, nx - 1) - 1
    iy = np.clip((x[:, 1] / f4(cell) + f4(1)).astype(np.int64), 1, ny - 1) - 1
    speed = np.sqrt(v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1])
    cnt, top = np.zeros((ny, nx)), [np.zeros((ny, nx), f4), np.zeros((ny, nx), f4)]
    tot = [np.zeros((ny, nx)), np.zeros((ny, nx))]
    for oy in (0, 1):
        for ox in (0, 1):
            at = (iy + oy, ix + ox)
            np.add.at(cnt, at, 2)  # sampled twice
            for k, q in enumerate((h, speed)):
                np.maximum.at(top[k], at, q)
                np.add.at(tot[k], at, 2.0 * q.astype(np.float64))
    sim.hazard_reset()
    sim.hazard_sample()
    sim.hazard_sample()
    np.testing.assert_array_equal(sim.raster(gfsph.RASTER_COUNT), cnt.astype(f4))
    np.testing.assert_array_equal(sim.raster(gfsph.RASTER_MAX_DEPTH), top[0])
    np.testing.assert_array_equal(sim.raster(gfsph.RASTER_MAX_VEL), top[1])
    np.testing.assert_allclose(sim.raster(gfsph.RASTER_SUM_DEPTH), tot[0].astype(f4), rtol=2.0 ** -23)
    np.testing.assert_allclose(sim.raster(gfsph.RASTER_SUM_VEL), tot[1].astype(f4), rtol=2.0 ** -23)
    # the raster on caller's buffers adds the same terms
    xd, hd = torch.from_numpy(x).cuda(), torch.from_numpy(h).cuda()
    out = torch.empty((ny, nx), device="cuda")
    st = gfsph.lib().gfsph_raster_idw_noalloc(n, C.c_void_p(xd.data_ptr()), C.c_void_p(hd.data_ptr()), None, nx, ny,
                                               0.0, 0.0, cell, cell, C.c_void_p(out.data_ptr()), None)
    torch.cuda.synchronize()
    assert st == 0
    np.testing.assert_allclose(out.cpu().numpy(), want, rtol=2.0 ** -23)
