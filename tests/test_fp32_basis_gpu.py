"""Krylov bases of more than 32 directions in FP32, where a lane of the scalars'
warp holds a second coefficient.  An FP32 solve usually ends its basis before:
every inner solve asks for three digits at most.  One weakly damped sweep a level
as preconditioner keeps the residual above that for all 48 directions, so that the
iterations are those of one basis.  With coefficients 33 to 48 lost the residual
would stay at what 32 directions reach; it has to fall well below half of it, as in
FP64 (to an eighth), and be the one that the operator gives for the result."""
import numpy as np
import pytest

import mdz
import oracle
from test_multigrid_odd_gpu import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
def test_directions_beyond_the_warp(precision):
    g, f = _case(67, 46)
    rng = np.random.default_rng(7)
    F = [rng.standard_normal(g.size(c)) * (t == -1) for c, t in ((-1, g.BCu), (-2, g.BCv))]
    Fp = rng.standard_normal(g.size(1))
    F.append(Fp - Fp.mean())
    norm = np.sqrt(sum(np.sum(q * q) for q in F))
    rel = {}
    ctx = mdz.Context(g, 1, 1)
    ctx.set_solver_options(nu1=1, nu2=0, omega=0.3, restart=48)
    for m in (32, 48):
        s = f.struct()
        d = [np.zeros(g.size(c)) for c in (-1, -2, 1)]
        its, r = mdz.C.c_int(0), mdz.C.c_double(0)
        st = ctx.L.mdz_SolveStokesDefect(ctx.h, mdz.C.byref(s), 0, precision, mdz.C.c_double(1e-12), m,
                                         *[mdz._dptr(a) for a in (*F, *d)], mdz.C.byref(its), mdz.C.byref(r))
        assert st == 5 and its.value == m   # not converged: the call says so
        res = [a - b for a, b in zip(oracle.stokes_apply(g, f, 0, *d), F)]
        rel[m] = np.sqrt(sum(np.sum(q * q) for q in res)) / norm
        assert rel[m] > 1e-3 and abs(r.value - rel[m]) <= 1e-6 * rel[m]
    ctx.close()
    assert rel[48] < 0.4 * rel[32], rel
