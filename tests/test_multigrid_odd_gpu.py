"""Multigrid levels of grids whose cell counts become odd on the way down: the
coarse level rounds up, its far wall lies one fine cell outside the box.  Every
level is the Galerkin product P^T A P of the level above with that P, and the
defect solve agrees with a direct solve of the oracle's assembled operator."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

import mdz
import oracle_step
from mg_reference import stencil_matrix, unknown_maps, velocity_block

pytestmark = pytest.mark.gpu


def prolongation(nxf, nzf, nxc, nzc):
    """P of a coarse level of nxc x nzc vertices onto nxf x nzf (coarse line I at fine line 2 I)."""
    iuf, ivf, nf = unknown_maps(nxf, nzf)
    iuc, ivc, nc = unknown_maps(nxc, nzc)

    def node(i):      # node-centred direction: (coarse line, weight)
        return [(i // 2, 1.0)] if i % 2 == 0 else [(i // 2, 0.5), (i // 2 + 1, 0.5)]

    def cell(j, n):   # cell-centred lines 1..n, the ghost lines mirrored
        j0 = (j - 1) // 2 + 1
        j1 = j0 + 1 if (j - 1) % 2 else j0 - 1
        return [(j0, 0.75), (j1, 0.25)] if 1 <= j1 <= n else [(j0, 1.0)]
    rows, cols, vals = [], [], []
    for fine, coarse, wx, wz in ((iuf, iuc, node, lambda j: cell(j, nzc - 1)), (ivf, ivc, lambda i: cell(i, nxc - 1), node)):
        for l, k in zip(*np.nonzero(fine >= 0)):
            for i, a in wx(k):
                for j, b in wz(l):
                    if coarse[j, i] >= 0:
                        rows.append(fine[l, k]); cols.append(coarse[j, i]); vals.append(a * b)
    return sp.csr_matrix((vals, (rows, cols)), shape=(nf, nc))


def _case(Nx, Nz):
    g = mdz.Grid(Nx, Nz, -0.5 * (Nx - 1) / (Nz - 1), 0.5 * (Nx - 1) / (Nz - 1), -0.5, 0.5).set_bc_pureshear(1.0)

    def eta(X, Z):
        return np.where(np.hypot(*np.meshgrid(X - 0.1, Z + 0.05)) < 0.2, 100.0, 1.0).ravel()
    f = mdz.GridFields(g, 1)
    f["eta_n"], f["eta_s"] = eta(g.xc, g.zc), eta(g.xg, g.zg)
    f["D11_n"], f["D22_n"], f["D33_s"] = 2 * f["eta_n"], 2 * f["eta_n"], f["eta_s"]
    return g, f


# odd cell counts at the first, second and third level, in one direction and in both
SIZES = [(26, 26), (31, 25), (51, 35), (67, 46), (101, 51), (77, 75)]


@pytest.mark.parametrize("Nx,Nz", SIZES)
@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 2e-6)])
def test_odd_levels_are_galerkin_products(Nx, Nz, precision, tol):
    g, f = _case(Nx, Nz)
    K, idx, n, n_p = oracle_step.assemble(g, f, 0)
    Fv = (np.sin(5 * g.zg)[:, None] * np.cos(3 * g.xvz)[None, :]).ravel() * (g.BCv == -1) * g.dx * g.dz
    ctx = mdz.Context(g, 1, 1)
    ctx.SolveStokesDefect(f, 0, precision, 1e-3, 300, np.zeros(g.size(-1)), Fv, np.zeros(g.size(1)))
    nl, nx, nz, su, sv = ctx.mg_stencils(precision, 0)
    A, _ = stencil_matrix(nx, nz, su, sv)
    assert spla.norm(A - velocity_block(g, K, idx)) < tol * spla.norm(A)
    odd = 0
    for level in range(1, nl):
        _, cx, cz, suc, svc = ctx.mg_stencils(precision, level)
        assert (cx - 1, cz - 1) == (nx // 2, nz // 2)   # cells: (n + 1) / 2 of the finer count
        odd += nx % 2 == 0 or nz % 2 == 0
        Ac, dropped = stencil_matrix(cx, cz, suc, svc)
        assert dropped == 0.0
        P = prolongation(nx, nz, cx, cz)
        assert spla.norm(Ac - P.T @ A @ P) < tol * spla.norm(Ac), level
        A, nx, nz = Ac, cx, cz
    assert odd > 0
    ctx.close()


@pytest.mark.parametrize("Nx,Nz", SIZES)
def test_defect_solve_on_odd_grids(Nx, Nz):
    g, f = _case(Nx, Nz)
    rng = np.random.default_rng(Nx)
    F = [rng.standard_normal(g.size(c)) * (t == -1) for c, t in ((-1, g.BCu), (-2, g.BCv))] + [np.zeros(g.size(1))]
    ctx = mdz.Context(g, 1, 1)
    du, dv, dp, its, rel = ctx.SolveStokesDefect(f, 0, 64, 1e-11, 500, *F)
    ctx.close()
    assert rel <= 1e-11 and its < 150
    want = oracle_step.solve_defect(g, f, 0, np.concatenate(F))
    nu, nv = g.size(-1), g.size(-2)
    for got, ref in ((du, want[:nu]), (dv, want[nu:nu + nv])):
        assert np.linalg.norm(got - ref) < 1e-8 * np.linalg.norm(ref)
    wp = want[nu + nv:]
    assert np.linalg.norm(dp - dp.mean() - (wp - wp.mean())) < 1e-8 * np.linalg.norm(wp - wp.mean())
