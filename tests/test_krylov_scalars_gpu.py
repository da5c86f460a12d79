"""The Krylov iteration's scalars, one warp with two coefficients per lane: bases
of 12, 31, 33 and 48 directions (several bases in a row, across the lanes' second
coefficient, the largest), run long enough to fill them, in both precisions.
The residual that the operator gives for the result is the one asked for; the
running norm may be off by the loss of orthogonality, hence the factor 3."""
import numpy as np
import pytest

import mdz
import oracle
from test_multigrid_odd_gpu import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("restart", [12, 31, 33, 48])
def test_basis_sizes(restart, precision):
    g, f = _case(67, 46)
    rng = np.random.default_rng(7)
    F = [rng.standard_normal(g.size(c)) * (t == -1) for c, t in ((-1, g.BCu), (-2, g.BCv))]
    Fp = rng.standard_normal(g.size(1))
    F.append(Fp - Fp.mean())
    rtol = 1e-9
    ctx = mdz.Context(g, 1, 1)
    ctx.set_solver_options(restart=restart)
    du, dv, dp, its, rel = ctx.SolveStokesDefect(f, 0, precision, rtol, 3000, *F)
    again = ctx.SolveStokesDefect(f, 0, precision, rtol, 3000, *F)
    ctx.close()
    assert rel <= rtol and (its > 48 or precision == 32)   # (FP32: the basis starts anew at each refinement)
    assert again[3] == its and np.array_equal(again[0], du) and np.array_equal(again[2], dp)   # fixed-order sums
    r = [a - b for a, b in zip(oracle.stokes_apply(g, f, 0, du, dv, dp), F)]
    assert np.sqrt(sum(np.sum(q * q) for q in r)) <= 3 * rtol * np.sqrt(sum(np.sum(q * q) for q in F))
