"""The V-cycle's launches against a CPU restatement of the same V-cycle: the
velocity block of one preconditioner application, recovered from a defect solve
stopped after its first Krylov vector, on grids around the sizes where a level
changes kernel (tile sizes, the one-CTA bottom, the dense coarsest level)."""
import numpy as np
import pytest
import scipy.sparse.linalg as spla

import mdz
import oracle
from mg_reference import stencil_matrix, unknown_maps
from test_multigrid_odd_gpu import _case, prolongation

pytestmark = pytest.mark.gpu


def vcycle(levels, f, nu1, nu2, omega, l=0):
    A, P = levels[l]
    if P is None:
        return spla.spsolve(A.tocsc(), f)
    d = A.diagonal()
    x = omega * f / d
    for _ in range(nu1 - 1):
        x = x + omega * (f - A @ x) / d
    x = x + P @ vcycle(levels, P.T @ (f - A @ x), nu1, nu2, omega, l + 1)
    for _ in range(nu2):
        x = x + omega * (f - A @ x) / d
    return x


# 21..: dense below the viscous level; 33, 49, 65 bottom from level 1 (FP32) or 2;
# 129, 201, 385: tile kernels of all three sizes; odd counts on several levels
SIZES = [(21, 21), (33, 17), (49, 33), (65, 65), (78, 53), (129, 65), (201, 127), (385, 257)]


@pytest.mark.parametrize("nu1,nu2", [(2, 1), (1, 2), (3, 0)])
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("Nx,Nz", SIZES)
def test_first_krylov_direction(Nx, Nz, precision, nu1, nu2):
    if (nu1, nu2) != (2, 1) and Nx > 150:
        pytest.skip("sweep counts at the small sizes")
    g, f = _case(Nx, Nz)
    rng = np.random.default_rng(Nx)
    F = [rng.standard_normal(g.size(c)) * (t == -1) for c, t in ((-1, g.BCu), (-2, g.BCv))]
    Fp = rng.standard_normal(g.size(1))
    Fp -= Fp.mean()
    ctx = mdz.Context(g, 1, 1)
    ctx.set_solver_options(nu1=nu1, nu2=nu2)
    s = f.struct()
    du, dv, dp = np.zeros(g.size(-1)), np.zeros(g.size(-2)), np.zeros(g.size(1))
    its, rel = mdz.C.c_int(0), mdz.C.c_double(0)
    st = ctx.L.mdz_SolveStokesDefect(ctx.h, mdz.C.byref(s), 0, precision, mdz.C.c_double(1e-30), 1,
                                     *[mdz._dptr(a) for a in (F[0], F[1], Fp, du, dv, dp)], mdz.C.byref(its), mdz.C.byref(rel))
    assert st == 5 and its.value == 1   # one iteration does not reach 1e-30: the call says so
    levels, dims = [], []
    nl = ctx.mg_stencils(precision, 0)[0]
    for level in range(nl):
        _, nx, nz, su, sv = ctx.mg_stencils(precision, level)
        dims.append((nx, nz))
        levels.append([stencil_matrix(nx, nz, su, sv)[0], None])
    for level in range(nl - 1):
        levels[level][1] = prolongation(*dims[level], *dims[level + 1])
    ctx.close()
    # the preconditioner on r0: zp = eta / celvol Fp, z = V-cycle(Fvel - B zp)
    zp = f["eta_n"] / (g.dx * g.dz) * Fp
    B = oracle.stokes_apply(g, f, 0, np.zeros(g.size(-1)), np.zeros(g.size(-2)), zp)
    iu, iv, n = unknown_maps(Nx, Nz)
    r = np.zeros(n)
    for m, a, b in ((iu, F[0], B[0]), (iv, F[1], B[1])):
        r[m[m >= 0]] = (a - b).reshape(m.shape)[m >= 0]
    z = vcycle(levels, r, nu1, nu2, 0.7)
    zu, zv = np.zeros(g.size(-1)), np.zeros(g.size(-2))
    zu.reshape(iu.shape)[iu >= 0], zv.reshape(iv.shape)[iv >= 0] = z[iu[iu >= 0]], z[iv[iv >= 0]]
    # the first iterate is the multiple of z that minimises the residual
    w = np.concatenate(oracle.stokes_apply(g, f, 0, zu, zv, zp - zp.mean()))
    a = w @ np.concatenate([F[0], F[1], Fp]) / (w @ w)
    tol = 1e-9 if precision == 64 else 2e-4   # sums of ~1e4 terms and a 1e2 contrast: 1e3..1e4 roundings
    for got, want in ((du, a * zu), (dv, a * zv), (dp - dp.mean(), a * (zp - zp.mean()))):
        assert np.linalg.norm(got - want) < tol * np.linalg.norm(want)
