"""FP32 evaluations of the local rheology: the FP64 solve takes over where the
FP32 one did not converge, also where its iterations ran out with finite
numbers."""
import ctypes as C
import os

import numpy as np
import pytest

import mdz
import mdz_build
import oracle
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
