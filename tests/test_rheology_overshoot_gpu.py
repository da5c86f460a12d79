"""Dislocation creep beside grain-boundary sliding.  The reference's local Newton
iteration leaves the sliding out of its slope, so with exponents above the sliding's
own an update can overshoot to a negative viscosity, from where it returns,
oscillates or runs away; with integer exponents every power is a number all the same
and the limited result is finite.  GPU against the oracle on rates over six
decades: finite wherever the oracle is, and equal where 1e-12 of the rates moves the
oracle by at most 1e-7.  Nodes where the power law is below 1e-8 of the rate at the
start are compared for finiteness only: the first residual, rate - sliding - power
law, is then the rounding of the first two (1e-16), and with it the first update."""
import numpy as np
import pytest

import mdz
import oracle

pytestmark = pytest.mark.gpu

KEYS = ("eta_n", "eta_s", "sxxd", "szzd", "eII_pwl", "exx_diss")


def _fields(g, scale):
    f = mdz.GridFields(g, 1)
    for node, s in ((1, ""), (0, "_s")):
        E = np.logspace(-3, 3, g.size(node)) * scale
        f["exxd" + s], f["ezzd" + s] = E, -E
    for k in ("T", "T_s", "mu_n", "mu_s", "bet_n", "bet_s", "d0_n", "d0_s"):
        f[k] = np.ones_like(f[k])
    f["C_n"], f["C_s"] = np.full(g.size(1), 1e20), np.full(g.size(0), 1e20)
    f["phase_perc_n"], f["phase_perc_s"] = np.ones((1, g.size(1))), np.ones((1, g.size(0)))
    return f


@pytest.mark.parametrize("n,ngbs,Agbs", [(3.0, 1.0, 0.1), (4.0, 1.0, 10.0), (4.0, 2.0, 1.0), (5.0, 2.0, 0.1), (3.0, 3.0, 1.0)])
def test_overshoot(n, ngbs, Agbs):
    g = mdz.Grid(66, 33, -1.0, 1.0, -0.5, 0.5).set_bc_pureshear(1.0)
    mat = mdz.Materials.from_phases([dict(pwlv=1, npwl=n, Apwl=1.0, fpwl=1.0, Fpwl=1.0, pref_pwl=1.0, gbsv=1, ngbs=ngbs,
                                          Agbs=Agbs, fgbs=1.0, Fgbs=1.0, rho=1.0, Slim=1e30, n_vp=1.0, gs_ref=1.0)], R=1.0)
    prm = mdz.RheoParams.make(dt=1.0, iselastic=0, step=1, mineta=1e-3, maxeta=1e3)
    ref = []
    for scale in (1.0, 1.0 + 1e-12, 1.0 - 1e-12):
        ref.append(_fields(g, scale))
        oracle.viscosity_grid(g, mat, prm, ref[-1])
    f = _fields(g, 1.0)
    ctx = mdz.Context(g, 1, 1)
    ctx.NonNewtonianViscosityGrid(mat, prm, f)
    ctx.close()
    for k in KEYS:
        a, b, c = (r[k] for r in ref)
        assert np.isfinite(a).all() and np.isfinite(f[k]).all(), k
        same = np.maximum(np.abs(a - b), np.abs(a - c)) <= 1e-7 * np.abs(a)
        E = np.logspace(-3, 3, len(a))
        eta_pwl, eta_gbs = E ** (1 / n - 1), Agbs ** (-1 / ngbs) * E ** (1 / ngbs - 1)
        same &= np.minimum(1.0, eta_gbs / eta_pwl) ** n > 1e-8
        assert same.mean() > 0.6, (k, same.mean())
        np.testing.assert_allclose(f[k][same], a[same], rtol=1e-6, err_msg=k)
