"""The fused search and density where its grouping can go wrong: the edges of
a block's particles and of the lanes-per-particle rule, neighbour lists longer
than the shared lists (repeated scans) and than the table, coincident
particles, clamped edge cells, more coarse particles than the direct scan
takes.  Sets are exact; densities and forces carry FP64 sums of the oracle's
FP32 terms in another order, so one rounding to FP32 separates them (1e-6)."""
import numpy as np
import pytest

import gfsph
import workloads

pytestmark = pytest.mark.gpu


def cloud(n, seed, box, hs, far=0, far_hs=1.0):
    rng = np.random.default_rng(seed)
    x = rng.uniform(5.0, 5.0 + box, (n, 2)).astype(np.float32)
    h = (hs * rng.uniform(0.8, 1.25, n)).astype(np.float32)
    if far:
        h[rng.choice(n, far, replace=False)] = np.float32(far_hs)
    return x, h


def check(oracle_mod, x, hs, forces=True, **opts):
    n = len(x)
    rng = np.random.default_rng(n)
    rho = rng.uniform(0.5, 1.5, n).astype(np.float32)
    mass = (rho * hs * hs * np.float32(0.25)).astype(np.float32)
    z = np.zeros((64, 64), np.float32)
    p = gfsph.make_params(workloads.voellmy_const(0.2, 500.0), pa_sph=2, nnps=2, sle=1, skf=opts.pop("skf", 1),
                          average_velocity=1, ic_adapt=0, h_inf=0.01, dt=0.01, dem_deriv=1, **opts)
    sim = gfsph.Sim(p, z, dx=20.0, dy=20.0)
    sim.upload(x, np.zeros_like(x), rho, mass, hs)
    dens = sim.density()
    off, idx = sim.neighbours()
    ref = oracle_mod.pairs(oracle_mod.MODE_FP32_DACC, p, x, hs, mass=mass, rho=rho, want_rho=True, want_force=forces)
    assert np.array_equal(off, ref["offsets"]) and np.array_equal(idx, ref["idx"])
    assert np.max(np.abs(dens - ref["rho"]) / np.abs(ref["rho"])) <= 1e-6
    if forces:
        f = sim.internal_forces()
        assert np.abs(f - ref["force"]).max() <= 1e-6 * max(np.abs(ref["force"]).max(), 1e-6)
    sim.close()


@pytest.mark.parametrize("skf", [1, 3])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 33, 128, 129, 11999, 12000, 12001])
def test_sets_and_density_at_group_edges(gfsph_lib, oracle_mod, n, skf):
    x, h = cloud(n, n, max(2.0, 0.6 * np.sqrt(n)), 1.0)
    check(oracle_mod, x, h, skf=skf)


@pytest.mark.parametrize("n", [99999, 100001])
def test_sets_where_two_lanes_begin(gfsph_lib, oracle_mod, n):
    x, h = cloud(n, n, 900.0, 2.2)
    check(oracle_mod, x, h, forces=False)


@pytest.mark.parametrize("n,box", [(160, 0.5), (600, 0.5), (600, 3.0)])
def test_lists_longer_than_the_shared_ones(gfsph_lib, oracle_mod, n, box):
    """Every particle near every other: each lane finds several lists' worth."""
    x, h = cloud(n, 3, box, 1.0)
    check(oracle_mod, x, h, max_neighbours=8)


def test_long_lists_with_two_lanes(gfsph_lib, oracle_mod):
    x, h = cloud(100500, 4, 900.0, 2.0)
    x[:700] = np.float32(450.0) + (x[:700] - np.float32(5.0)) / np.float32(450.0)
    check(oracle_mod, x, h, forces=False)


def test_coincident_particles(gfsph_lib, oracle_mod):
    x, h = cloud(300, 5, 12.0, 1.0)
    x[100:150] = x[:50]
    check(oracle_mod, x, h)


@pytest.mark.parametrize("far,hs", [(1, 9.0), (40, 12.0), (130, 30.0)])
def test_coarse_particles_by_direct_scan(gfsph_lib, oracle_mod, far, hs):
    x, h = cloud(9000, 6, 120.0, 1.0, far, hs)
    check(oracle_mod, x, h)


def test_more_coarse_particles_than_the_direct_scan(gfsph_lib, oracle_mod):
    x, h = cloud(60000, 7, 1100.0, 1.0, 4500, 7.0)
    check(oracle_mod, x, h, forces=False)


@pytest.mark.parametrize("n", [44999, 45001])
def test_sets_and_forces_where_lanes_change(gfsph_lib, oracle_mod, n):
    x, h = cloud(n, n, 500.0, 1.8)
    check(oracle_mod, x, h)
