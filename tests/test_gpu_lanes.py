"""The pair kernels on either side of each change in the lanes per particle (8 below 12,000 particles, 4 below 45,000, 2
below 500,000, then 1; the adjoint's four lanes up to 100,000) against the oracle: internal forces and one step of the
plain, the staged (normalised density) and the soil-and-water form, and the adjoint.  The tolerances are those of the
same comparisons on small cases: the lanes change the order of FP64 sums of FP32 terms only."""
import numpy as np
import pytest

import gfsph
import workloads

pytestmark = pytest.mark.gpu
EDGES = [11_999, 12_000, 44_999, 45_000, 499_999, 500_000]


def channel(n):
    w = workloads.fractal_channel(n_target=int(n * 1.03), dem_k=8 if n < 20_000 else 10, cell=5.0, erosion=None)
    assert w.n >= n
    rng = np.random.default_rng(n)
    jit = (1.0 + rng.uniform(-0.05, 0.05, n)).astype(np.float32)
    return w, w.x[:n], w.v[:n] + np.float32(0.5) * (jit - 1)[:, None], w.rho[:n] * jit, w.mass[:n] * jit, w.hsml[:n]


def close(got, ref, keys, tol=1e-6):
    for k in keys:
        r = getattr(ref, k).astype(np.float64)
        err = np.abs(got[k] - r) / np.maximum(np.abs(r), 1e-3)
        assert err.max() <= tol, (k, err.max())


@pytest.mark.parametrize("n", EDGES)
@pytest.mark.parametrize("opts", [{}, {"nor_density": 1}])
def test_step_and_forces(gfsph_lib, oracle_mod, n, opts):
    w, x, v, rho, mass, hsml = channel(n)
    p = workloads.make_params(w, gfsph, ic_adapt=0, sle=1, **opts)
    topol = oracle_mod.initial_topol(w.z, w.dx, w.dy, w.const, deriv=p.dem_deriv, mode=oracle_mod.MODE_FP32)
    sim = gfsph.Sim(p, w.z, dx=w.dx, dy=w.dy, topol=topol.astype(np.float32))
    sim.upload(x, v, rho, mass, hsml)
    f = sim.internal_forces()
    if not opts:
        ref = oracle_mod.pairs(oracle_mod.MODE_FP32_DACC, p, x, hsml, mass=mass, rho=rho, want_sets=False, want_rho=True,
                               want_force=True)["force"]
        assert np.abs(f - ref).max() <= 1e-6 * np.abs(ref).max()
    sim.upload(x, v, rho, mass, hsml)
    sim.step(1)
    got = sim.download()
    sim.close()
    ny, nx = w.z.shape
    st = oracle_mod.State(x, v, rho, mass, hsml, topol, dt=p.dt)
    oracle_mod.run(oracle_mod.MODE_FP32_DACC, p, nx, ny, w.dx, w.dy, st, 1)
    assert np.array_equal(got["flag"], st.flag)
    close(got, st, ("x", "v", "rho", "hsml"))


@pytest.mark.parametrize("n", EDGES[:4] + [120_000])
def test_soil_and_water_step(gfsph_lib, oracle_mod, n):
    w, a = workloads.soil_and_pond(spacing=0.75 * np.sqrt(37_329.0 / (n * 1.02)), scale=2.0)
    drop = len(a["rho"]) - n
    assert 0 <= drop < n // 10
    a = {k: q[drop:] for k, q in a.items()}  # soil first: some of it is left out, all of the water stays
    p = workloads.make_params(w, gfsph)
    sim = gfsph.Sim(p, w.z, dx=w.dx, dy=w.dy)
    sim.upload(a["x"], a["v"], a["rho"], a["mass"], a["hsml"], itype=a["itype"])
    sim.step(1)
    got = sim.download()
    sim.close()
    ny, nx = w.z.shape
    topol = oracle_mod.initial_topol(w.z, w.dx, w.dy, w.const, deriv=p.dem_deriv)
    flag = np.where(a["itype"] == 2, 2, 0).astype(np.int32)
    st = oracle_mod.State(a["x"], a["v"], a["rho"], a["mass"], a["hsml"], topol, flag=flag, dt=p.dt)
    oracle_mod.run(oracle_mod.MODE_FP32_DACC, p, nx, ny, w.dx, w.dy, st, 1)
    assert np.array_equal(got["flag"], st.flag & 1)
    for k in ("x", "v", "rho", "hsml"):
        ref = getattr(st, k).astype(np.float32)
        assert np.abs(got[k] - ref).max() <= 1e-6 * max(np.abs(ref).max(), 1.0), k


@pytest.mark.parametrize("n", [11_999, 12_000, 99_999, 100_000, 500_000])
def test_adjoint(gfsph_lib, oracle_mod, n):
    """Three steps, recorded at every second, against the exact derivative of the device's own single-precision
    trajectory along the friction, the volumes, the positions and the velocities, 2e-5 of the direction's terms."""
    w, x, v, rho, mass, hsml = channel(n)
    v = v + np.float32([0.1, 3.0])
    p = workloads.make_params(w, gfsph, sle=0, ic_adapt=0, dt=0.02)
    topol = oracle_mod.initial_topol(w.z, w.dx, w.dy, w.const, deriv=p.dem_deriv, mode=oracle_mod.MODE_FP32)
    rng = np.random.default_rng(n)
    gx, gv = rng.normal(size=(2, n, 2)).astype(np.float32)
    gh = rng.normal(size=n).astype(np.float32)
    sim = gfsph.Sim(p, w.z, dx=w.dx, dy=w.dy, topol=topol.astype(np.float32))
    sim.upload(x, v, rho, mass, hsml)
    adj = gfsph.Adjoint(sim, 3, every=2)
    g = adj.backward(gx, gv, gh)
    adj.close()
    sim.close()
    ny, nx = w.z.shape
    st0 = oracle_mod.State(x, v, rho, mass, hsml, topol, dt=p.dt)
    dm, dx0, dv0 = rng.normal(size=n) * mass, rng.normal(size=(n, 2)), rng.normal(size=(n, 2))
    both = dict(seed_m=dm, seed_x=dx0, seed_v=dv0)
    terms = [g["mass"] * dm, (g["x0"] * dx0).ravel(), (g["v0"] * dv0).ravel()]
    for seed, got, scale in ((dict(seed_mu=1.0), g["tanfi"], abs(g["tanfi"])),
                             (both, sum(float(t.sum()) for t in terms), sum(float(np.abs(t).sum()) for t in terms))):
        _, _, _, dx, dv, dh = oracle_mod.tangent(p, nx, ny, w.dx, w.dy, st0, 3, single=True, **seed)
        ref = float((gx * dx).sum() + (gv * dv).sum() + (gh * dh).sum())
        assert abs(got - ref) <= 2e-5 * scale, (list(seed), got, ref, scale)
