"""FP32 evaluations of the local rheology: the FP64 solve takes over where the
FP32 one did not converge, also where its iterations ran out with finite
numbers; and the material options whose constants the host forms per precision
(grain-size, melt and pressure dependence, non-linear diffusion creep and
regularisation) agree with FP64 to FP32's tolerance."""
import ctypes as C
import os

import numpy as np
import pytest

import mdz
import mdz_build
import mdz_setups
import oracle
from test_rheology_options_gpu import VARIANTS
from test_rheology_overshoot_gpu import _fields

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("native") / "viscosity_probe.so")
    mdz_build._run([mdz_build._nvcc()] + mdz_build.NVCC_FLAGS + [
        "-shared", "-o", so, os.path.join(HERE, "native", "viscosity_probe.cu"), "-L" + mdz_build.LIBDIR, "-lmdoodz_gb300",
        "-Xlinker", "-rpath," + mdz_build.LIBDIR])
    mdz.load_library()
    L = C.CDLL(so)

    def run(ctx, mat, prm, f, fp32):
        s = f.struct()
        assert L.probe_viscosity(ctx.h, C.byref(mat), C.byref(prm), C.byref(s), fp32) == 0
    return run


def _residual(E, n, ngbs, Agbs, real):
    """The last relative residual of the plain iteration in precision `real`."""
    E = np.asarray(E, real)
    n, ngbs, two = real(n), real(ngbs), real(2)
    B = real(Agbs) ** (real(-1) / ngbs)
    C1, Cg = two ** -n, (two * B) ** -ngbs
    eta = np.minimum(E ** (real(1) / n - real(1)), B * E ** (real(1) / ngbs - real(1)))
    with np.errstate(all="ignore"):
        for _ in range(20):
            T = two * eta * E
            pwl, r = C1 * T ** n, E - C1 * T ** n - Cg * T ** ngbs
            res = np.abs(r / E)
            eta = np.where(res < 1e-6, eta, eta + r / (pwl * n / eta))
    return res


@pytest.mark.parametrize("n,ngbs,Agbs", [(3.0, 1.0, 0.1), (4.0, 2.0, 1.0), (5.0, 2.0, 0.1)])
def test_fp64_takes_over_exhausted_solves(probe, n, ngbs, Agbs):
    g = mdz.Grid(66, 33, -1.0, 1.0, -0.5, 0.5).set_bc_pureshear(1.0)
    mat = mdz.Materials.from_phases([dict(pwlv=1, npwl=n, Apwl=1.0, fpwl=1.0, Fpwl=1.0, pref_pwl=1.0, gbsv=1, ngbs=ngbs,
                                          Agbs=Agbs, fgbs=1.0, Fgbs=1.0, rho=1.0, Slim=1e30, n_vp=1.0, gs_ref=1.0)], R=1.0)
    prm = mdz.RheoParams.make(dt=1.0, iselastic=0, step=1, mineta=1e-3, maxeta=1e3)
    ref = []
    for scale in (1.0, 1.0 + 1e-12, 1.0 - 1e-12):
        ref.append(_fields(g, scale))
        oracle.viscosity_grid(g, mat, prm, ref[-1])
    f = [_fields(g, 1.0), _fields(g, 1.0)]
    ctx = mdz.Context(g, 1, 1)
    for fp32 in (0, 1):
        probe(ctx, mat, prm, f[fp32], fp32)
    ctx.close()
    E = np.logspace(-3, 3, g.size(1))
    a, b, c = (r["sxxd"] for r in ref)
    # far from converged in both precisions, and an FP64 result that 1e-12 of the rates moves by at most 1e-7
    out = (_residual(E, n, ngbs, Agbs, np.float64) > 1e-2) & (_residual(E, n, ngbs, Agbs, np.float32) > 1e-2)
    out &= np.maximum(np.abs(a - b), np.abs(a - c)) <= 1e-7 * np.abs(a)
    assert out.sum() > 30
    np.testing.assert_allclose(f[1]["sxxd"][out], f[0]["sxxd"][out], rtol=1e-6)


@pytest.mark.parametrize("name", sorted(VARIANTS))
def test_options_in_fp32(probe, name):
    """The FP32 loops stop at 1e-6 of the rate and at 1e-4 of the yield function
    (absolute or relative), for stresses of about 1: fields to 1e-3 of their largest
    value, ten times that.  A wrong constant moves them by its own relative error."""
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
    o = oracle.Oracle(g, 3)
    o.set_markers(x, z, (rng.random(len(x)) * 3).astype(np.int32))
    phases = [dict(p, **{k: v for k, v in change.items()
                         if not (k.endswith("lin") and not p.get("linv")) and not (k.endswith("pwl") and not p.get("pwlv"))})
              for p in RHEO_PHASES]
    mat = mdz.Materials.from_phases(phases, R=RHEO_R)
    prm = mdz.RheoParams.make(**dict(RHEO_MODEL, **model))
    f = mdz.GridFields(g, 3, ins)
    f["phase_perc_n"] = o.P2Mastah(np.zeros(3), None, g.tags(1), 0, 0, 1, 1, 1)
    f["phase_perc_s"] = o.P2Mastah(np.zeros(3), None, g.tags(0), 0, 0, 1, 0, 1)
    for k, n in (("sxxd0_s", 0), ("szzd0_s", 0), ("sxz0_n", 1)):
        f[k] = rng.normal(size=g.size(n)) * 0.3
    oracle.strain_rates(g, f)
    got = []
    ctx = mdz.Context(g, 3, 1)
    for fp32 in (0, 1):
        h = mdz.GridFields(g, 3, {k: v.copy() for k, v in f.a.items()})
        probe(ctx, mat, prm, h, fp32)
        got.append(h)
    ctx.close()
    for k in ("eta_n", "eta_s", "sxxd", "szzd", "sxz", "eII_pwl", "eII_lin", "eII_pl", "exx_diss"):
        a, b = got[0][k], got[1][k]
        assert np.abs(a - b).max() <= 1e-3 * np.abs(a).max(), (k, np.abs(a - b).max() / np.abs(a).max())
    assert np.any(got[0]["sxxd"] != got[1]["sxxd"])   # FP32 it was
