"""gfsph_internal_forces with two materials: pairs of a soil and a water particle (marked in the neighbour table) take
no part, so either material's forces are those it has alone."""
import numpy as np
import pytest

import gfsph
import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("material", [1, 2])
def test_each_material_as_if_alone(gfsph_lib, material):
    w, a = workloads.soil_and_pond()

    def forces(keep):
        sim = gfsph.Sim(gfsph.make_params(w.const, sle=1, ic_adapt=0, dt=0.01, ws_interact=1, sw_alg=0), w.z, dx=w.dx,
                        dy=w.dy)
        sim.upload(*(a[k][keep] for k in ("x", "v", "rho", "mass", "hsml")), itype=a["itype"][keep])
        f = sim.internal_forces()
        sim.close()
        return f

    own = a["itype"] == material
    both, alone = forces(np.ones(len(own), bool))[own], forces(own)
    # sums of the same FP32 terms in FP64, in another order: the last place of the FP32 result
    assert np.abs(alone).max() > 0.0
    assert np.abs(both - alone).max() <= 1e-6 * np.abs(alone).max()
