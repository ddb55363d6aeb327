"""The persistent CG with its rows in memory (above 303,104 dofs, two rows a thread of 148 blocks of 1024) and the last
sizes with rows in registers, on fields that differ from node to node, without and with prescribed dofs (the masked
product).  The right-hand side is the assembled matrix times a known x, so that x is the solution; tol is on squared
norms, so the relative error is about sqrt(tol) times the condition number of the mass matrix (16), plus FP32."""
import numpy as np
import pytest

import gfsph
import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,ndofn", [(592, 512, 1), (553, 549, 1), (401, 390, 2), (296, 512, 2)])
@pytest.mark.parametrize("fixed", [False, True])
def test_known_solution(gfsph_lib, nx, ny, ndofn, fixed):
    im, co = workloads.p1_mesh(nx, ny, 2.0)
    m = workloads.p1_mass_matrices(im, co).astype(np.float32)
    g = np.zeros((len(im), 3 * ndofn, 3 * ndofn), np.float32)
    for d in range(ndofn):  # unconnected components: assembled zeros
        g[:, d::ndofn, d::ndofn] = m * np.float32(1 + d)
    n = nx * ny * ndofn
    rng = np.random.default_rng(nx + ndofn)
    ref = (np.sin(0.37 * np.arange(n)) + 0.5 * rng.standard_normal(n)).astype(np.float32)
    dof = ((im - 1)[:, :, None] * ndofn + np.arange(ndofn)).reshape(len(im), -1)
    b = np.zeros(n)
    np.add.at(b, dof, np.einsum("eij,ej->ei", g.astype(np.float64), ref[dof].astype(np.float64)))
    fix, val = np.zeros(n, np.int32), np.zeros(n, np.float32)
    if fixed:
        at = rng.choice(n, n // 9, replace=False)
        fix[at] = 1
        val[at] = ref[at]
    cg = gfsph.CG(im, g, ndofn)
    x, _, _, it = cg.solve(b.astype(np.float32), fix, val, tol=1e-12)
    cg.close()
    assert it >= 1
    assert np.linalg.norm(x - ref) <= 3e-5 * np.linalg.norm(ref)
    assert np.abs(x - ref).max() <= 1e-3
