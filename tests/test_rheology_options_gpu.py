"""Local rheology with the material options that take other branches of the
solve than the standard materials: non-linear diffusion creep and viscoplastic
regularisation, grain-size, melt and pressure dependence, dilation, elasticity
off, step 0; GPU against the oracle node by node, and the learned start's
polish against the plain solve."""
import numpy as np
import pytest

import mdz
import mdz_setups
import oracle
from test_oracle_rheology import _check

pytestmark = pytest.mark.gpu

TOL = 1e-10   # as the rheology parity tests: local Newton tolerance 1e-13, tangents a few hundred times that
KEYS = ("eta_n", "eta_s", "eta_phys_n", "eta_phys_s", "VE_n", "sxxd", "szzd", "sxz", "eII_el", "eII_pl", "eII_pwl", "eII_lin",
        "eII_cst", "d_n", "exx_el", "exx_diss", "exz_diss", "detadexx_n", "detadezz_n", "detadgxz_n", "detadp_n", "detadgxz_s",
        "detadp_s", "ddivpdexx_n", "ddivpdp_n", "p_corr", "div_u_el", "div_u_pl", "Wtot", "Wdiss", "OverS_n", "OverS_s")

VARIANTS = {
    "plain": ({}, {}),
    "lin_nonlinear": (dict(nlin=2.0), {}),
    "lin_grain_size": (dict(mlin=2.0, gs_ref=0.7), {}),
    "lin_nonlinear_grain_melt": (dict(nlin=1.5, mlin=1.0, gs_ref=0.7, alin=0.3, rlin=1.2, flin=2.0, Vlin=0.04), {}),
    "pwl_grain_melt": (dict(mpwl=1.0, apwl=0.4, rpwl=1.2, fpwl=2.0, Vpwl=0.03, gs_ref=1.3), {}),
    "vp_nonlinear": (dict(n_vp=3.0, eta_vp=0.05), {}),
    "dilation": (dict(eta_vp=0.03), dict(dil=0.1)),
    "no_plasticity_cap": (dict(Slim=0.2), {}),
    "inelastic": ({}, dict(iselastic=0)),
    "step0": ({}, dict(step=0)),
    "clamped": ({}, dict(mineta=0.05, maxeta=0.4, clamp_tangent=1)),
    "geometric": (dict(nlin=2.0), dict(eta_avg=2)),
}


@pytest.mark.parametrize("name", sorted(VARIANTS))
def test_option_vs_oracle(name):
    from golden.make_golden import RHEO_MODEL, RHEO_PHASES, RHEO_R, rheology_inputs
    change, model = VARIANTS[name]
    model = dict(model)
    dil = model.pop("dil", 0.0)
    g = mdz.Grid(70, 37, -1.0, 1.0, -0.5, 0.5).set_bc_pureshear(1.0)
    rng = np.random.default_rng(11)
    ins = rheology_inputs(g, rng)
    ins["phi0_n"] = 0.1 * rng.random(g.size(1))
    ins["d0_n"] = 0.8 + 0.4 * rng.random(g.size(1))
    ins["dil_n"], ins["dil_s"] = np.full(g.size(1), dil), np.full(g.size(0), dil)
    ins["p0_n"] = 0.5 * rng.random(g.size(1))
    x, z = mdz_setups.seed_markers(g, 3, 3, 0.5, 9)
    ph = (rng.random(len(x)) * 3).astype(np.int32)
    o = oracle.Oracle(g, 3)
    o.set_markers(x, z, ph)
    phases = [dict(p, **{k: v for k, v in change.items()
                         if not (k.endswith("lin") and not p.get("linv")) and not (k.endswith("pwl") and not p.get("pwlv"))})
              for p in RHEO_PHASES]
    mat = mdz.Materials.from_phases(phases, R=RHEO_R)
    prm = mdz.RheoParams.make(**dict(RHEO_MODEL, **model))
    fo = mdz.GridFields(g, 3, ins)
    fo["phase_perc_n"] = o.P2Mastah(np.zeros(3), None, g.tags(1), 0, 0, 1, 1, 1)
    fo["phase_perc_s"] = o.P2Mastah(np.zeros(3), None, g.tags(0), 0, 0, 1, 0, 1)
    for k, n in (("sxxd0_s", 0), ("szzd0_s", 0), ("sxz0_n", 1)):
        fo[k] = rng.normal(size=g.size(n)) * 0.3
    fg = mdz.GridFields(g, 3, dict(fo.a))
    oracle.strain_rates(g, fo)
    oracle.viscosity_grid(g, mat, prm, fo)
    ctx = mdz.Context(g, 3, 1)
    ctx.StrainRateComponents(fg)
    ctx.NonNewtonianViscosityGrid(mat, prm, fg)
    ctx.close()
    for k in KEYS:
        _check(fg[k], fo[k], k, TOL)
