"""Launches that need several CTAs at once (a cooperative grid, a cluster) may be
refused where the device, or the part of it that the process has, cannot hold
them.  The library is built a second time with the runtime's calls replaced
by such answers (native/fake_runtime.h): the calls go on by launches without that
need and agree with the oracle."""
import os

import pytest

import mdz
import mdz_build
import test_thermal_one_launch_gpu as thermal

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


@pytest.fixture(scope="module")
def refused(tmp_path_factory):
    """mdz on the library whose launches are refused."""
    so = _variant(tmp_path_factory.mktemp("refused"), "refused", ["thermal"], "-DFAKE_REFUSED_LAUNCHES")
    kept, mdz._lib = mdz._lib, None
    try:
        yield mdz.load_library(so)
    finally:
        mdz._lib = kept


@pytest.mark.parametrize("Nx,Nz", [(5, 4), (33, 9), (130, 259)])
def test_energy_step_without_cooperative_launch(refused, Nx, Nz):
    thermal.test_energy_step_sizes(Nx, Nz)
