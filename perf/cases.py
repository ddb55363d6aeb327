"""The work a user of gfsph has it do, as cases that can be timed.

Every case goes through the package's public entry points (gfsph.Sim,
gfsph.Ensemble, gfsph.Adjoint, gfsph.Gfl) on seeded synthetic inputs.  Most of
them are plot intervals of a run, as the reference's time loop and gfsph_run
take them: the particle state from host buffers, the steps of the interval,
the outputs of that plot time, the state back in host buffers.

Two kinds of particle states are met in a run and both are here: the release,
all particles at rest on a lattice with one smoothing length ("release"), and
the flow some seconds later ("flow"): stretched along the channel, unordered,
moving, with smoothing lengths that follow 2 sqrt(m/h) and a thin front of
isolated particles whose smoothing lengths are many times the mean.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deslizamientos-y-flujos_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import gfsph  # noqa: E402
import workloads  # noqa: E402


def listed():
    return [
        # the smallest calls: launches and latency count.  A gully slide at the size of the reference's own
        # example (frictional with v^2/R curvature, pore pressure icpwp 3, nnps 4, adaptive dt)
        dict(name="gully_850", kind="steps", scene="gully", n=850, state="release", steps=40, dem_k=8, cell=10.0),
        # the granular collapse on the inclined plane (Voellmy, fixed dt)
        dict(name="plane_2k", kind="steps", scene="plane", n=1941, state="release", steps=40),
        # a mid-size debris flow under way, odd count: erosion, levels of smoothing lengths, coarse particles
        dict(name="channel_flow_23k", kind="steps", scene="channel", n=23_003, state="flow", steps=25, dem_k=9,
             cell=5.0),
        # the benchmark's release: 200k particles, Voellmy with Hungr erosion, adaptive dt
        dict(name="channel_release_200k", kind="steps", scene="channel", n=200_000, state="release", steps=20,
             dem_k=10, cell=5.0),
        # the same flow later in its run
        dict(name="channel_flow_200k", kind="steps", scene="channel", n=200_000, state="flow", steps=20, dem_k=10,
             cell=5.0),
        # the largest: four releases kilometres apart (block-sparse cell grid), Bingham
        dict(name="releases_1m", kind="steps", scene="releases", n=1_000_000, state="release", steps=10, dem_k=11,
             cell=4.0),
        # stage-dependent pressure: normalised density, terrain-normal gravity, pore pressure (staged RK45)
        dict(name="staged_60k", kind="steps", scene="staged", n=60_000, state="flow", steps=10, dem_k=9, cell=5.0),
        # soil and water particles
        dict(name="pond_37k", kind="steps", scene="pond", n=37_000, state="release", steps=10),
        # hazard realizations of ragged size advanced together, exceedance raster
        dict(name="ensemble_10", kind="ensemble", members=10, n=12_000, steps=16, dem_k=9, cell=5.0),
        # back-analysis: forward record, raster misfit, adjoint sweep
        dict(name="calibration_50k", kind="calibration", n=50_000, steps=20, every=5, law="voellmy", dem_k=9,
             cell=5.0),
        # the water mesh of the coupled run: Taylor-Galerkin steps on 498k triangles
        dict(name="water_mesh_250k", kind="mesh", nx=500, ny=500, steps=20, nfric=1),
        # the coupling pass: soil depth and its gradient on a mesh window, consistent mass matrix by CG
        dict(name="coupling_300", kind="coupling", n=100_000, window=300, dem_k=10, cell=2.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps"] * 8 + ["ensemble", "calibration", "mesh", "coupling"])
    if kind == "steps":
        scene = rng.choice(["gully", "plane", "channel", "channel", "channel", "releases", "staged", "pond"])
        if scene == "plane":
            return dict(kind=kind, scene=scene, n=_log(rng, 500, 20_000), state="release", steps=rng.randint(10, 40))
        if scene == "gully":
            return dict(kind=kind, scene=scene, n=_log(rng, 300, 60_000), state=rng.choice(["release", "flow"]),
                        steps=rng.randint(10, 30), dem_k=rng.choice([7, 8, 9]), cell=10.0)
        if scene == "channel":
            return dict(kind=kind, scene=scene, n=_log(rng, 900, 400_000), state=rng.choice(["release", "flow"]),
                        steps=rng.randint(8, 20), dem_k=rng.choice([9, 10]), cell=5.0)
        if scene == "releases":
            return dict(kind=kind, scene=scene, n=_log(rng, 20_000, 700_000), state="release",
                        steps=rng.randint(5, 10), dem_k=11, cell=rng.choice([2.0, 4.0]))
        if scene == "staged":
            return dict(kind=kind, scene=scene, n=_log(rng, 1_000, 100_000), state=rng.choice(["release", "flow"]),
                        steps=rng.randint(4, 12), dem_k=9, cell=5.0)
        return dict(kind=kind, scene=scene, n=_log(rng, 2_000, 60_000), state="release", steps=rng.randint(4, 12))
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(3, 12), n=_log(rng, 2_000, 20_000), steps=rng.randint(8, 16),
                    dem_k=rng.choice([8, 9]), cell=5.0)
    if kind == "calibration":
        steps = rng.randint(6, 20)
        return dict(kind=kind, n=_log(rng, 2_000, 60_000), steps=steps, every=rng.randint(1, steps),
                    law=rng.choice(["voellmy", "bingham"]), dem_k=rng.choice([8, 9]), cell=5.0)
    if kind == "mesh":
        return dict(kind=kind, nx=_log(rng, 60, 500), ny=_log(rng, 60, 500), steps=rng.randint(5, 20),
                    nfric=rng.choice([0, 1, 4, 5]))
    return dict(kind=kind, n=_log(rng, 5_000, 150_000), window=_log(rng, 60, 320), dem_k=10, cell=2.0)


# ------------------------------------------------------------------ inputs

def _pinned(a, dtype=np.float32):
    """A copy in page-locked host memory, as a program that moves it every interval keeps it."""
    t = torch.from_numpy(np.ascontiguousarray(a, dtype=dtype).copy())
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


def _flowing(x, rho, mass, rng, spacing):
    """A release some seconds into its flow: stretched and spread towards +y, jittered, moving, the depth thinned
    by the stretch, a front of isolated particles; smoothing lengths 2 sqrt(m/h)."""
    n = x.shape[0]
    y0, y1 = float(x[:, 1].min()), float(x[:, 1].max())
    xc = 0.5 * float(x[:, 0].min() + x[:, 0].max())
    s = (x[:, 1] - y0) / (y1 - y0)
    wide = 1.0 + 0.25 * s
    px = xc + (x[:, 0] - xc) * wide
    py = y0 + (y1 - y0) * (s + 0.6 * s * s)
    h = rho / (wide * (1.0 + 1.2 * s))
    front = rng.random(n) < 0.001
    px = px + rng.uniform(-0.3, 0.3, n) * spacing
    py = py + rng.uniform(-0.3, 0.3, n) * spacing
    px = np.where(front, xc + rng.normal(0.0, 0.15 * (y1 - y0), n), px)
    py = np.where(front, y0 + 1.6 * (y1 - y0) + rng.exponential(0.1 * (y1 - y0), n), py)
    h = np.where(front, h * rng.uniform(0.005, 0.1, n), h)
    v = np.stack([0.4 * (px - xc) / (y1 - y0) + rng.normal(0, 0.05, n), 4.0 + 6.0 * s + rng.normal(0, 0.05, n)], 1)
    return np.stack([px, py], 1).astype(np.float32), v.astype(np.float32), h.astype(np.float32), \
        (2.0 * np.sqrt(mass / h)).astype(np.float32)


_GULLY = {1: 9.8, 2: 2000.0, 3: 300.0, 5: 7, 9: 0.6, 10: 0.01, 13: 0.001, 14: 1.0, 15: 0.01}
_STAGED = {1: 9.8, 2: 2000.0, 3: 400.0, 5: 5, 9: 0.3, 10: 0.01, 13: 0.001, 14: 1.0, 15: 0.01, 16: 1}


def _scene(case, seed):
    """(const, options, z, cell, state arrays, itype) of a `steps` case."""
    scene, n = case["scene"], case["n"]
    rng = np.random.default_rng(seed)
    s = int(rng.integers(1, 1 << 30))
    if scene == "plane":
        w = workloads.inclined_plane(seed=s, spacing=2.0 * math.sqrt(1941.0 / n))
    elif scene == "releases":
        w = workloads.multi_release(n_target=n, dem_k=case["dem_k"], cell=case["cell"], seed=s)
    elif scene == "pond":
        w, a = workloads.soil_and_pond(spacing=0.75 * math.sqrt(37_329.0 / n), scale=2.0)
        jit = (1.0 + rng.uniform(-0.01, 0.01, len(a["rho"]))).astype(np.float32)
        arr = dict(x=a["x"], v=a["v"], rho=a["rho"] * jit, mass=a["mass"] * jit, hsml=a["hsml"])
        return w.const, w.options, w.z, w.dx, arr, a["itype"]
    else:
        w = workloads.fractal_channel(n_target=n, dem_k=case["dem_k"], cell=case["cell"], seed=s,
                                      erosion=(0.005, 2.0) if scene == "channel" else None)
    const, opts = dict(w.const), dict(w.options)
    if scene == "gully":
        const, opts = dict(_GULLY), dict(opts, nnps=4, icpwp=3, pwp0rel=1.0)
    elif scene == "staged":
        const, opts = dict(_STAGED), dict(opts, nor_density=1, icpwp=3, pwp0rel=0.3)
    x, v, rho, mass, hsml = w.x, w.v, w.rho, w.mass, w.hsml
    if case["state"] == "flow":
        x, v, rho, hsml = _flowing(x.astype(np.float64), rho.astype(np.float64), mass.astype(np.float64), rng,
                                   float(w.meta["lattice"]))
    return const, opts, w.z, w.dx, dict(x=x, v=v, rho=rho, mass=mass, hsml=hsml), None


def _out_buffers(n):
    return dict(x=_pinned(np.zeros((n, 2))), v=_pinned(np.zeros((n, 2))), rho=_pinned(np.zeros(n)),
                mass=_pinned(np.zeros(n)), hsml=_pinned(np.zeros(n)), flag=_pinned(np.zeros(n), np.int32))


def _mesh_inputs(case, seed):
    rng = np.random.default_rng(seed)
    nx, ny, d = case["nx"], case["ny"], 5.0
    intmat, coord = workloads.p1_mesh(nx, ny, d)
    x, y = coord[:, 0] / (nx * d), coord[:, 1] / (ny * d)
    z = 20.0 * (1.0 - y) + rng.uniform(1, 3) * np.cos(6.0 * x + rng.uniform(0, 6)) * np.cos(5.0 * y)
    h = 1.0 + 0.5 * np.cos(9.0 * x + rng.uniform(0, 6)) * np.cos(8.0 * y) + 0.05 * rng.random(len(x))
    u = np.stack([h, 0.2 * h * np.sin(7 * x), h * (0.5 + 0.1 * np.cos(6 * y))], 1)
    const = {1: 9.8, 2: 1000.0, 3: 0.03, 5: case["nfric"], 6: 50.0, 7: 10.0, 9: 0.05, 10: 0.01}
    return intmat, coord, z.astype(np.float32), u.astype(np.float32), const


# ------------------------------------------------------------------ a user's program

def prepare(case, seed):
    kind = case["kind"]
    if kind == "mesh":
        intmat, coord, z, u, const = _mesh_inputs(case, seed)
        return dict(case=case, g=gfsph.Gfl(coord, intmat, z, const, ntype=3, ngaus=3, niter=3), u=_pinned(u))
    if kind == "steps":
        const, opts, z, cell, a, itype = _scene(case, seed)
        sim = gfsph.Sim(gfsph.make_params(const, **opts), z, dx=cell, dy=cell)
        n = a["x"].shape[0]
        return dict(case=case, sim=sim, a={k: _pinned(v) for k, v in a.items()}, dt=opts["dt"],
                    itype=None if itype is None else _pinned(itype, np.int32), out=_out_buffers(n),
                    pwp=bool(opts.get("icpwp")))
    rng = np.random.default_rng(seed)
    s = int(rng.integers(1, 1 << 30))
    if kind == "ensemble":
        ws, z = [], None
        for k in range(case["members"]):  # ragged: 0.2 to 2 times n particles; friction sampled per realization
            f = 0.2 + 1.8 * ((0.618034 * (k + 1)) % 1.0)
            ws.append(workloads.fractal_channel(n_target=int(case["n"] * f), dem_k=case["dem_k"], cell=case["cell"],
                                                seed=s, mu=float(rng.uniform(0.08, 0.30)), mean_depth=4.0 * f,
                                                xi=float(np.exp(rng.normal(math.log(400.0), 0.3))), z=z))
            z = ws[0].z
        e = gfsph.Ensemble([workloads.make_params(w, gfsph) for w in ws], ws[0].z, dx=ws[0].dx, dy=ws[0].dy)
        ins = [{k: _pinned(getattr(w, k)) for k in ("x", "v", "rho", "mass", "hsml")} for w in ws]
        return dict(case=case, e=e, ins=ins, outs=[_out_buffers(w.n) for w in ws], dt=0.01)
    w = workloads.fractal_channel(n_target=case["n"], dem_k=case["dem_k"], cell=case["cell"], seed=s, erosion=None)
    const, opts = dict(w.const), dict(w.options, ic_adapt=0, sle=0, dt=0.02)
    if case.get("law") == "bingham":
        const = {1: 9.8, 2: 2000.0, 5: 4, 6: 800.0, 7: 40.0, 10: 0.01, 15: 0.01}
    sim = gfsph.Sim(gfsph.make_params(const, **opts), w.z, dx=w.dx, dy=w.dy)
    v = (w.v + np.array([0.1, 3.0], np.float32) * (1 + 0.01 * rng.standard_normal((w.n, 1)))).astype(np.float32)
    a = {k: _pinned(q) for k, q in dict(x=w.x, v=v, rho=w.rho, mass=w.mass, hsml=w.hsml).items()}
    if kind == "calibration":
        target = np.maximum(0.0, 2.0 + rng.standard_normal(w.z.shape)).astype(np.float32)
        return dict(case=case, sim=sim, a=a, target=_pinned(target), zeros=_pinned(np.zeros((w.n, 2))), dt=0.02)
    sim.upload(a["x"], a["v"], a["rho"], a["mass"], a["hsml"])  # coupling: the soil as its run has left it
    nx, k = w.z.shape[1], case["window"]
    y0 = int(0.137 * nx) - k // 2
    return dict(case=case, sim=sim, x0=nx // 2 - k // 2, y0=max(y0, 0))


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "mesh":
        g = st["g"]
        g.set_state(st["u"])
        g.step(case["steps"], 0.02)
        u, t = g.state()
        return dict(u=u, t=t)
    if kind == "ensemble":
        e = st["e"]
        for m, a in zip(e.members, st["ins"]):
            m.upload(a["x"], a["v"], a["rho"], a["mass"], a["hsml"])
            m.set_time(0.0, st["dt"])
        e.step(case["steps"])
        e.sample()
        prob = e.exceedance(1.0)
        outs = [m.download(out=o) for m, o in zip(e.members, st["outs"])]
        return dict(prob=prob, x=[o["x"] for o in outs], v=[o["v"] for o in outs], rho=[o["rho"] for o in outs],
                    mass=[o["mass"] for o in outs], hsml=[o["hsml"] for o in outs])
    sim = st["sim"]
    if kind == "coupling":
        hs, g = sim.gradhs(st["x0"], st["y0"], case["window"], case["window"], niter=0, tol=1e-10)
        return dict(hs=hs, g=g)
    a = st["a"]
    sim.upload(a["x"], a["v"], a["rho"], a["mass"], a["hsml"], itype=st.get("itype"))
    sim.set_time(0.0, st["dt"])
    if kind == "calibration":
        adj = gfsph.Adjoint(sim, case["steps"], case["every"])
        loss, gx, gh = sim.raster_misfit(st["target"])
        grad = adj.backward(gx, st["zeros"], gh)
        adj.close()
        return dict(loss=loss, gx=gx, gh=gh, x0=grad["x0"], v0=grad["v0"], mass=grad["mass"], tanfi=grad["tanfi"],
                    xi=grad["xi"], tauy=grad["tauy"])
    _, t, done = sim.step(case["steps"])
    out = dict(sim.download(out=st["out"]), t=t, done=done)
    if case["scene"] in ("channel", "gully"):  # plot time: the hazard statistics and the depth raster
        sim.hazard_reset()
        sim.hazard_sample()
        out["depth"] = sim.raster(gfsph.RASTER_DEPTH_IDW)
        out["max_v"] = sim.raster(gfsph.RASTER_MAX_VEL)
    if st["pwp"]:
        out["pwp"] = sim.pwp()
    return out


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    """Bytes each pass has to move and operations it has to do.  Per particle-step 168 B (the state and the packed
    fields read and written once per phase) and ~48 neighbours; per pair the kernel value and gradient (~35
    operations), the pressure term (~8) and the velocity average (~10); per particle four stages of the basal law
    (~80 each)."""
    kind = case["kind"]

    def step(n, staged=False):
        return dict(bytes=(168.0 + (3 * 60.0 if staged else 0.0)) * n,
                    flops=n * (48 * ((35.0 + 8 + 10) if not staged else (35.0 + 4 * 8 + 10 + 5 * 4)) + 4 * 80.0))

    if kind == "steps":
        n, k = case["n"], case["steps"]
        s = step(n, case["scene"] in ("staged", "pond"))
        return dict(bytes=k * s["bytes"] + 68.0 * n, flops=k * s["flops"])
    if kind == "ensemble":
        n, k = 1.1 * case["n"] * case["members"], case["steps"]
        s = step(n)
        return dict(bytes=k * s["bytes"] + 68.0 * n, flops=k * s["flops"])
    if kind == "calibration":
        n, k = case["n"], case["steps"]
        s = step(n)  # the forward step, the replayed step, and the reverse of its pair sums and stages
        return dict(bytes=k * 3 * s["bytes"], flops=k * (2 * s["flops"] + n * (48 * 120.0 + 4 * 200.0)))
    if kind == "mesh":
        npo, ne = case["nx"] * case["ny"], 2 * (case["nx"] - 1) * (case["ny"] - 1)
        return dict(bytes=case["steps"] * (npo * (12.0 + 36 + 36 + 12 * 6) + ne * (12.0 + 28 + 36)),
                    flops=case["steps"] * (npo * 120.0 + ne * (3 * 90.0 + 2 * 40.0)))
    n, nn = case["n"], case["window"] ** 2
    its = 12
    return dict(bytes=16.0 * n + nn * 12.0 + its * 2 * nn * (7 * 12.0 + 7 * 8.0), flops=its * 2 * nn * 26.0)


# ------------------------------------------------------------------ the same in 64 bits

def exact(case, seed):
    """The Voellmy and Bingham runs (plane, channel, releases) in 64-bit torch; None for the other options."""
    if case["kind"] != "steps" or case["scene"] not in ("plane", "channel", "releases"):
        return None
    const, opts, z, cell, a, _ = _scene(case, seed)
    return _Exact(const, opts, z, cell, a).run(case)


class _Exact:
    """Depth-integrated SPH with summation density, the cubic spline, RK4, Voellmy or Bingham friction, Hungr
    erosion, the smoothing-length update and the velocity average, in 64 bits."""

    def __init__(self, const, opts, z, cell, a):
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        f = lambda q: torch.from_numpy(np.asarray(q, np.float64)).to(dev)  # noqa: E731
        c32 = {k: float(np.float32(v)) for k, v in const.items()}
        self.c, self.o, self.cell = c32, opts, float(np.float32(cell))
        self.hinf = float(np.float32(opts["h_inf"]))
        self.x, self.v, self.h, self.m, self.hs = (f(a[k]) for k in ("x", "v", "rho", "mass", "hsml"))
        zz = f(np.asarray(z, np.float32))
        self.ny, self.nx = zz.shape
        gx, gy = torch.zeros_like(zz), torch.zeros_like(zz)
        gx[1:-1, 1:-1] = (zz[1:-1, 2:] - zz[1:-1, :-2]) / (2 * self.cell)
        gy[1:-1, 1:-1] = (zz[2:, 1:-1] - zz[:-2, 1:-1]) / (2 * self.cell)
        self.gx, self.gy = gx.reshape(-1), gy.reshape(-1)

    def pairs(self):
        """Every (i, j), i != j, with |x_i - x_j| < h_i + h_j."""
        x, hs = self.x, self.hs
        lev = torch.floor(torch.log2(hs / hs.min())).long()
        ii, jj = [], []
        groups = [(torch.nonzero(lev == k)[:, 0]) for k in torch.unique(lev).tolist()]
        for b in groups:
            for a in groups:
                c = float(hs[a].max() + hs[b].max()) * 1.000001
                lo = x.min(0).values - 2 * c
                nx = int(float((x[:, 0].max() - lo[0]) / c)) + 4
                kb = torch.floor((x[b] - lo) / c).long()
                keys, order = torch.sort(kb[:, 1] * nx + kb[:, 0])
                ka = torch.floor((x[a] - lo) / c).long()
                for dy in (-1, 0, 1):
                    base = (ka[:, 1] + dy) * nx + ka[:, 0]
                    s, e = torch.searchsorted(keys, base - 1), torch.searchsorted(keys, base + 2)
                    cnt = e - s
                    i = torch.repeat_interleave(torch.arange(len(a), device=x.device), cnt)
                    off = torch.arange(len(i), device=x.device) - torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt, cnt)
                    j = b[order[s[i] + off]]
                    i = a[i]
                    d = x[i] - x[j]
                    keep = ((d * d).sum(1) < (hs[i] + hs[j]) ** 2) & (i != j)
                    ii.append(i[keep])
                    jj.append(j[keep])
        return torch.cat(ii), torch.cat(jj)

    def slopes(self, x):
        c = self.cell
        ix = (x[:, 0] / c).floor().clamp(0, self.nx - 2)
        iy = (x[:, 1] / c).floor().clamp(0, self.ny - 2)
        a, b = x[:, 0] / c - ix, x[:, 1] / c - iy
        n1 = (iy * self.nx + ix).long()

        def at(g):
            return (1 - a) * (1 - b) * g[n1] + a * (1 - b) * g[n1 + 1] + a * b * g[n1 + 1 + self.nx] + (1 - a) * b * g[n1 + self.nx]

        return at(self.gx), at(self.gy)

    def friction(self, x, v, h):
        """Gravity, basal friction over h, and the erosion rate, before the reversal filter."""
        c = self.c
        g, comp = c[1], c[15]
        wet = h >= comp
        hh = torch.where(wet, h, torch.full_like(h, comp))
        hu, hv = torch.where(wet, h * v[:, 0], 0.0), torch.where(wet, h * v[:, 1], 0.0)
        hinv = torch.where(wet, 1.0 / hh, 0.0)
        hvm = torch.sqrt(hu * hu + hv * hv)
        vmod = hvm * hinv
        hvi = torch.where(hvm >= 1e-5, 1.0 / hvm.clamp(min=1e-30), 0.0)
        hf = hh.clamp(min=c[10])
        zx, zy = self.slopes(x)
        if int(c[5]) == 4:
            ah = 6.0 * c[7] * hvm / (c[6] * hf * hf)
            b2 = -(32.0 * ah) - 114.0
            xh = (-b2 - torch.sqrt(b2 * b2 - 4.0 * 48.0 * 65.0)) / 96.0
            k = torch.where(ah > 50.0, 3.0 * c[7] / c[2] / (hf * hf),
                            torch.where(ah < 0.01, c[6] / c[2] * hvi, c[6] / xh / c[2] * hvi))
            fx, fy, rest = k * hu, k * hv, torch.zeros_like(h)
            tot = torch.sqrt(fx * fx + fy * fy)
            rest = tot
        else:
            cf = torch.full_like(h, max(g * c[9], 0.0))
            vmod = torch.sqrt((v * v).sum(1))
            fx = cf * hu * hvi * hh + g * vmod * v[:, 0] / c[3]
            fy = cf * hv * hvi * hh + g * vmod * v[:, 1] / c[3]
            rest = cf
        er = c.get(22, 0.0) * hh * vmod if c.get(21, 0.0) > 0 else torch.zeros_like(h)
        return hh, hinv, vmod, -g * zx, -g * zy, fx, fy, rest, er

    def ext(self, x, v, h, fin, dt):
        hh, hinv, vmod, gx, gy, fx, fy, rest, er = self.friction(x, v, h)
        a0, a1 = gx + fin[:, 0], gy + fin[:, 1]
        d0, d1 = -fx * hinv, -fy * hinv
        vs0, vs1 = v[:, 0] + dt * (a0 + d0), v[:, 1] + dt * (a1 + d1)
        vm = vmod.clamp(min=1e-30)
        t0, t1 = v[:, 0] / vm, v[:, 1] / vm
        rev = (vs0 * v[:, 0] + vs1 * v[:, 1] < 0) & ((a0 * t0 + a1 * t1) * (d0 * t0 + d1 * t1) < 0)
        mx = torch.where(rev, (v[:, 0] / dt + a0) * hh, fx)
        my = torch.where(rev, (v[:, 1] / dt + a1) * hh, fy)
        am = torch.sqrt(a0 * a0 + a1 * a1)
        s0, s1 = rest * a0 / am.clamp(min=1e-30), rest * a1 / am.clamp(min=1e-30)
        hold = am <= torch.sqrt(s0 * s0 + s1 * s1)
        s0, s1 = torch.where(hold, a0, s0), torch.where(hold, a1, s1)
        s0, s1 = torch.where(am > 1e-5, s0, 0.0) * hh, torch.where(am > 1e-5, s1, 0.0) * hh
        move = vmod > 1e-5
        fx, fy = torch.where(move, mx, s0), torch.where(move, my, s1)
        e0 = gx - fx / hh - er * v[:, 0] * hinv
        e1 = gy - fy / hh - er * v[:, 1] * hinv
        return torch.stack([e0, e1], 1)

    def step(self, dt):
        c, o = self.c, self.o
        if o["ic_adapt"] == 1:
            dtm = float((self.hs / (3.0 * torch.sqrt(c[1] * self.h.clamp(min=self.hinf)).clamp(min=1e-6))).min())
            dt = dtm if dtm < dt else min(1.1 * dt, dtm)
        i, j = self.pairs()
        n = len(self.h)
        d = self.x[i] - self.x[j]
        r = torch.sqrt((d * d).sum(1))
        mh = 0.5 * (self.hs[i] + self.hs[j])
        q = r / mh
        fac = 15.0 / (7.0 * math.pi * mh * mh)
        u = (2.0 - q).clamp(min=0.0)
        w = torch.where(q <= 1.0, fac * (2.0 / 3.0 - q * q + 0.5 * q ** 3), fac / 6.0 * u ** 3)
        gr = torch.where(q <= 1.0, fac * (-2.0 + 1.5 * q) / (mh * mh), -0.5 * fac * u * u / (mh * r.clamp(min=1e-30)))
        zero = torch.zeros(n, dtype=torch.float64, device=self.x.device)
        w0 = 15.0 / (7.0 * math.pi * self.hs * self.hs) * (2.0 / 3.0)
        h = (w0 * self.m).index_add(0, i, self.m[j] * w)
        k = -c[1] * self.m[j] * gr
        fin = torch.stack([zero.index_add(0, i, k * d[:, 0]), zero.index_add(0, i, k * d[:, 1])], 1)
        hc = h.clamp(min=self.hinf)
        v, ex = self.v, torch.zeros_like(self.v)
        dx, dv = torch.zeros_like(v), torch.zeros_like(v)
        for s in range(4):
            f1, f2 = (0.0, 0.5, 0.5, 1.0)[s], (1.0, 2.0, 2.0, 1.0)[s]
            xs = self.x + f1 * dt * v
            v = self.v + f1 * dt * (ex + fin)
            ex = self.ext(xs, v, hc, fin, dt)
            dv = dv + f2 * (ex + fin)
            dx = dx + f2 * v
        self.x, self.v = self.x + dt / 6.0 * dx, self.v + dt / 6.0 * dv
        er = self.friction(self.x, self.v, h)[8]
        self.m = self.m + dt * er * self.m / h
        if o["sle"] == 1:
            self.hs = 2.0 * torch.sqrt(self.m / h)
        self.h = h
        if o["average_velocity"]:
            k = -0.6 * self.m[j] / (h[i] + h[j]) * w
            dv = self.v[i] - self.v[j]
            self.v = self.v + torch.stack([zero.index_add(0, i, k * dv[:, 0]), zero.index_add(0, i, k * dv[:, 1])], 1)
        return dt

    def raster(self):
        c, x = self.cell, self.x
        num = torch.zeros(self.nx * self.ny, dtype=torch.float64, device=x.device)
        den = torch.zeros_like(num)
        ix, iy = (x[:, 0] / c).floor().long(), (x[:, 1] / c).floor().long()
        for a in range(-1, 3):
            for b in range(-1, 3):
                px, py = ix + a, iy + b
                ok = (px >= 0) & (px < self.nx) & (py >= 0) & (py < self.ny)
                dist = torch.sqrt((x[:, 0] - px * c) ** 2 + (x[:, 1] - py * c) ** 2).clamp(min=1e-6) / (c * math.sqrt(2.0))
                at = (py * self.nx + px)[ok]
                num.index_add_(0, at, (self.h / dist)[ok])
                den.index_add_(0, at, (1.0 / dist)[ok])
        return torch.where(den >= 1e-6, num / den.clamp(min=1e-30), num).reshape(self.ny, self.nx)

    def run(self, case):
        dt, t = float(np.float32(self.o["dt"])), 0.0
        for _ in range(case["steps"]):
            dt = self.step(dt)
            t += dt
        out = dict(x=self.x, v=self.v, rho=self.h, mass=self.m, hsml=self.hs, flag=None, t=t, done=None)
        if case["scene"] == "channel":
            out["depth"], out["max_v"] = self.raster(), None
        return out
