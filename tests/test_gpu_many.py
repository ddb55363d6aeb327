"""k_density on either side of the particle count beyond which its launches get more blocks (24 rounds of 148 x 7 blocks of
128 threads, two lanes a particle), in both cell layouts: two releases out of each other's reach have the depths that
each has alone.  Each half is below the line; its pairs are the same, summed in FP64 in another order and rounded to FP32
once: an ulp at most."""
import numpy as np
import pytest

import gfsph
import workloads

pytestmark = pytest.mark.gpu
LINE = 24 * 148 * 7 * 128 // 2


def depths(x, rho):
    sim = gfsph.Sim(gfsph.make_params(workloads.voellmy_const(0.2, 500.0), pa_sph=2, nnps=2, sle=0, skf=1,
                                      average_velocity=1, ic_adapt=0, h_inf=0.01, dt=0.01, dem_deriv=1),
                    np.zeros((64, 64), np.float32), dx=100.0, dy=100.0)
    sim.upload(x, np.zeros_like(x), rho, rho.copy(), np.full(len(rho), 2.0, np.float32))
    r = sim.density()
    sim.close()
    return r


@pytest.mark.parametrize("apart", [30, 4400])  # m; at 4400 the box has too many cells for the dense layout
@pytest.mark.parametrize("n", [LINE, LINE + 1])
def test_two_releases_have_the_depths_of_each_alone(gfsph_lib, n, apart):
    m = (n + 1) // 2
    k = int(np.sqrt(m)) + 1
    g = np.stack(np.meshgrid(np.arange(k), np.arange(k)), -1).reshape(-1, 2).astype(np.float32)
    a, b = g[:m] + np.float32(40), g[:n - m] + np.float32(40 + k + apart)
    rho = np.random.default_rng(n).uniform(0.8, 1.2, n).astype(np.float32)
    both = depths(np.concatenate([a, b]), rho)
    alone = np.concatenate([depths(a, rho[:m]), depths(b, rho[m:])])
    assert both.min() > 0.1
    assert (np.abs(both - alone) <= np.spacing(alone)).all()
