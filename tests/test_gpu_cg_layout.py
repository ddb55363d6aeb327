"""The persistent CG where its layout and its branches can go wrong: dofs around
a warp of rows and a block, rows kept in registers and in memory, prescribed
dofs (the masked product), assembled zeros.  Against the dense solution of the
same system; tol is on squared norms, so the relative error is about
sqrt(tol) times the condition number of the mass matrix (16), plus FP32 output."""
import numpy as np
import pytest

import gfsph
import workloads

pytestmark = pytest.mark.gpu


def system(nx, ny, ndofn=1):
    im, co = workloads.p1_mesh(nx, ny, 2.0)
    m = workloads.p1_mass_matrices(im, co).astype(np.float32)
    if ndofn == 1:
        return im, m
    g = np.zeros((len(im), 3 * ndofn, 3 * ndofn), np.float32)  # unconnected components: assembled zeros
    for d in range(ndofn):
        g[:, d::ndofn, d::ndofn] = m
    return im, g


def dense(im, g, ndofn, n):
    K = np.zeros((n, n))
    dof = ((im - 1)[:, :, None] * ndofn + np.arange(ndofn)).reshape(len(im), -1)
    for e in range(len(im)):
        K[np.ix_(dof[e], dof[e])] += g[e].astype(np.float64)
    return K


@pytest.mark.parametrize("nx,ny,ndofn", [(2, 2, 1), (4, 8, 1), (3, 11, 1), (5, 13, 2), (32, 32, 1), (25, 41, 1),
                                         (23, 23, 2)])
@pytest.mark.parametrize("fixed", [False, True])
def test_solution_against_the_dense_one(gfsph_lib, nx, ny, ndofn, fixed):
    im, g = system(nx, ny, ndofn)
    n = nx * ny * ndofn
    rng = np.random.default_rng(nx * 100 + ny)
    b = rng.standard_normal(n).astype(np.float32)
    fix = np.zeros(n, np.int32)
    val = np.zeros(n, np.float32)
    if fixed:
        at = rng.choice(n, max(1, n // 7), replace=False)
        fix[at] = 1
        val[at] = rng.standard_normal(len(at)).astype(np.float32)
    cg = gfsph.CG(im, g, ndofn)
    x, _, _, it = cg.solve(b, fix, val, tol=1e-12)
    cg.close()
    K = dense(im, g, ndofn, n)
    free = fix == 0
    ref = val.astype(np.float64)
    ref[free] = np.linalg.solve(K[np.ix_(free, free)], b[free].astype(np.float64) - K[np.ix_(free, ~free)] @ ref[~free])
    assert it >= 1
    assert np.linalg.norm(x - ref) <= 3e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("nx", [551, 560])
def test_rows_in_registers_and_in_memory_agree(gfsph_lib, nx):
    """303,601 dofs keep their rows in memory (two rows a thread hold 303,104), 551 x 550 in registers: the same
    field, a solution known in closed form (M times a constant, the lumped masses)."""
    ny = 550 if nx == 551 else nx
    im, g = system(nx, ny)
    lump = np.zeros(nx * ny)
    np.add.at(lump, im - 1, g.astype(np.float64).sum(2))
    cg = gfsph.CG(im, g)
    x, _, _, _ = cg.solve((3.0 * lump).astype(np.float32), tol=1e-12)
    cg.close()
    assert np.abs(x - 3.0).max() <= 1e-4
