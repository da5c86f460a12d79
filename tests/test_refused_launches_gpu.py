"""Launches that need several CTAs at once (a cooperative grid, a cluster) may be
refused where the device, or the part of it that the process has, cannot hold
them.  The library is built a second time with the runtime's calls replaced
by such answers (native/fake_runtime.h): the calls go on by launches without that
need and agree with the oracle.  And a kernel's limit of shared memory, which
belongs to the process, does not depend on the call that sets it."""
import contextlib
import ctypes as C
import os

import pytest

import mdz
import mdz_build
import test_krylov_scalars_gpu as krylov
import test_thermal_one_launch_gpu as thermal
import test_vcycle_gpu as vcycle

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def _variant(tmp, name, sources, *flags):
    """The library with `sources` compiled behind native/fake_runtime.h."""
    objs = {os.path.basename(s)[:-3]: os.path.join(mdz_build.OBJ, os.path.basename(s)[:-3] + ".o")
            for s in sorted(mdz_build.glob.glob(os.path.join(mdz_build.CSRC, "*.cu")))}
    for s in sources:
        objs[s] = str(tmp / (s + ".o"))
        mdz_build._run([mdz_build._nvcc()] + mdz_build.NVCC_FLAGS + list(flags) + [
            "-include", os.path.join(HERE, "native", "fake_runtime.h"), "-c", os.path.join(mdz_build.CSRC, s + ".cu"),
            "-o", objs[s]])
    so = str(tmp / ("libmdoodz_%s.so" % name))
    mdz_build._run([mdz_build._nvcc()] + mdz_build.ARCH + ["-shared", "-o", so] + list(objs.values()) + ["-lcudart"])
    return so


@contextlib.contextmanager
def _loaded(so):
    """mdz on the library `so`."""
    kept, mdz._lib = mdz._lib, None
    try:
        yield mdz.load_library(so)
    finally:
        mdz._lib = kept


@pytest.fixture(scope="module")
def refused(tmp_path_factory):
    return _variant(tmp_path_factory.mktemp("refused"), "refused", ["thermal", "solver"], "-DFAKE_REFUSED_LAUNCHES")


@pytest.mark.parametrize("Nx,Nz", [(5, 4), (33, 9), (130, 259)])
def test_energy_step_without_cooperative_launch(refused, Nx, Nz):
    with _loaded(refused):
        thermal.test_energy_step_sizes(Nx, Nz)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("Nx,Nz", [(33, 17), (67, 46), (129, 65)])
def test_solve_without_clusters(refused, Nx, Nz, precision):
    """The V-cycle's levels as launches of their own: one application against the
    restatement of the cycle, and a solve whose residual the oracle confirms."""
    with _loaded(refused):
        vcycle.test_first_krylov_direction(Nx, Nz, precision, 2, 1)
        krylov.test_basis_sizes(33, precision)


def test_energy_step_sets_one_limit_for_all_grids(tmp_path):
    """(Another thread's call may set it between this one's setting and its launch.)"""
    with _loaded(_variant(tmp_path, "recorded", ["thermal"], "-DFAKE_RECORD_LIMITS")) as L:
        for Nx, Nz in ((17, 18), (402, 401), (33, 9)):
            thermal.test_energy_step_sizes(Nx, Nz)
        n = C.c_int()
        L.probe_limits_get.restype = C.POINTER(C.c_int)
        limits = L.probe_limits_get(C.byref(n))[:n.value]
    assert len(limits) == 6 and len(set(limits)) == 1, limits
