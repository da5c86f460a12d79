"""The V-cycle where its bottom, run by a cluster of eight CTAs, is widest or
emptiest: levels just below and above its limits of rows (2048 in FP64: 33 x 32
cells; 4096 in FP32: 45 x 46), levels with fewer rows than CTAs, long thin
levels, one to three sweeps on either side.  Against the CPU restatement, with
the tolerance of the other V-cycle tests."""
import pytest

from test_vcycle_gpu import test_first_krylov_direction as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu1,nu2", [(2, 1), (1, 3), (3, 0)])
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("Nx,Nz", [(9, 9), (11, 13), (17, 97), (65, 65), (67, 65), (67, 67), (91, 93), (93, 93)])
def test_bottom_of_the_vcycle(Nx, Nz, precision, nu1, nu2):
    if precision == 32 and Nx == 17:
        pytest.skip("the stiff inclusion spans the box: conditioned beyond FP32's tolerance here")
    check(Nx, Nz, precision, nu1, nu2)
