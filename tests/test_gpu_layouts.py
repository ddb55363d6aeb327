"""Runs that change between the dense and the block-sparse cell layout on one handle: the results are those of a handle
that has known nothing else, and the steps after a change take the time they take on such a handle."""
import numpy as np
import pytest

import gfsph
import workloads

pytestmark = pytest.mark.gpu
DENSE, SPARSE = 30.0, 5600.0  # m between the two halves of the release


def release(n, apart):
    """Two blocks of a lattice; kilometres apart the box holds more cells than the dense layout takes (4M, or 8 a particle)."""
    k = int(np.sqrt(n / 2)) + 1
    g = np.stack(np.meshgrid(np.arange(k), np.arange(k)), -1).reshape(-1, 2)[:(n + 1) // 2].astype(np.float64)
    x = np.concatenate([g + 40.0, g + 40.0 + (k + apart)])[:n].astype(np.float32)
    rng = np.random.default_rng(n)
    rho = rng.uniform(0.8, 1.2, n).astype(np.float32)
    return x, np.zeros_like(x), rho, rho.copy(), np.full(n, 2.0, np.float32)


def handle():
    return gfsph.Sim(gfsph.make_params(workloads.voellmy_const(0.2, 500.0), pa_sph=2, nnps=2, sle=0, skf=1,
                                       average_velocity=1, ic_adapt=0, h_inf=0.01, dt=0.01, dem_deriv=1),
                     np.zeros((64, 64), np.float32), dx=100.0, dy=100.0)


def go(sim, a, steps):
    sim.upload(*a)
    sim.set_time(0.0, 0.01)
    sim.step(steps)
    return sim.download()


@pytest.mark.parametrize("n", [900, 13_000, 60_000])
def test_results_across_the_layouts(gfsph_lib, n):
    sim = handle()
    for apart in (DENSE, SPARSE, SPARSE, DENSE, SPARSE):
        a = release(n, apart)
        got = go(sim, a, 5)
        fresh = handle()
        ref = go(fresh, a, 5)
        fresh.close()
        assert all(np.array_equal(got[k], ref[k]) for k in ref), apart
    sim.close()


@pytest.mark.parametrize("before,after", [(DENSE, SPARSE), (SPARSE, DENSE)])
def test_steps_after_a_change_are_not_slower(gfsph_lib, before, after):
    """Device time of the first batch after a change of layout against a batch that stays in it, the best of three each.
    Grids that followed the layout of earlier batches made it up to three times as long; the clocks and the rest of the
    box differ by far less than the half allowed."""
    n = 200_000
    sim = handle()
    states = {apart: release(n, apart) for apart in (before, after)}

    def batches(apart, count, steps):
        sim.upload(*states[apart])
        sim.set_time(0.0, 0.01)
        ms = []
        for _ in range(count):
            sim.profile(2)
            sim.step(steps)
            ms.append(sim.profile_read()["step_batches"][0])
            sim.profile(0)
        return ms

    for apart in (before, after):  # capacities grown
        batches(apart, 2, 1)
    changed, stays = [], []
    for _ in range(3):
        batches(before, 6, 1)
        changed += batches(after, 1, 8)
        batches(after, 6, 1)
        stays += batches(after, 1, 8)
    sim.close()
    assert min(changed) <= 1.5 * min(stays), (changed, stays)
