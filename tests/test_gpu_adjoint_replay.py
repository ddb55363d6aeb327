"""The backward sweep on a handle that no longer replays the recorded steps: uploaded with another size and back, so that
its neighbour table is as narrow as at the start again and a replayed step overflows it, or with search tunables that put
particles of the record on a coarse level.  Every checkpoint interval returns the error, whether a step fails where the
segment is recovered or where it is reversed, and the handle runs on afterwards."""
import numpy as np
import pytest

import gfsph
import workloads

pytestmark = pytest.mark.gpu
ERR_CAPACITY, ERR_UNSUPPORTED = -3, -4
NSTEPS = 5


def recorded(every, hsml=None, **opts):
    w = workloads.fractal_channel(n_target=1500, dem_k=8, cell=5.0, erosion=None)
    sim = gfsph.Sim(workloads.make_params(w, gfsph, sle=0, ic_adapt=0, **opts), w.z, dx=w.dx, dy=w.dy)
    a = [w.x, w.v, w.rho, w.mass, w.hsml if hsml is None else hsml(w)]
    sim.upload(*a)
    return sim, a, gfsph.Adjoint(sim, NSTEPS, every=every)


def refused(sim, a, adj, status):
    g = np.ones((len(a[0]), 2), np.float32)
    with pytest.raises(gfsph.GfsphError) as e:
        adj.backward(g, g)
    assert e.value.status == status
    adj.close()
    sim.upload(*a)
    assert sim.step(3)[2] == 3
    out = sim.download()
    assert all(np.isfinite(out[k]).all() for k in ("x", "v", "rho"))
    sim.close()


@pytest.mark.parametrize("every", [1, 2, NSTEPS])
def test_table_too_narrow_for_the_replay(gfsph_lib, every):
    sim, a, adj = recorded(every, max_neighbours=8)
    m = len(a[0]) - 40
    sim.upload(*(q[:m] for q in a))
    sim.upload(*a)
    refused(sim, a, adj, ERR_CAPACITY)


@pytest.mark.parametrize("every", [1, 2, NSTEPS])
def test_particles_coarse_under_other_tunables(gfsph_lib, every):
    def hsml(w):
        h = w.hsml.copy()
        h[::100] *= np.float32(2.5)  # regular up to twice 1.5 times the mean, coarse beyond twice the mean
        return h

    sim, a, adj = recorded(every, hsml)
    sim.set_search(1.0, 3.0)
    refused(sim, a, adj, ERR_UNSUPPORTED)
