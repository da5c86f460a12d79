"""FP32 inner products of the Krylov basis: the bound of their rounding.  A thread
adds its products up in FP32 before the block sums go to FP64, so the error of a
sum of positive products is at most (chain + 5 of the warp's shuffles + 1 of the
product) half units.  With a quarter of a first round of loads 1 and everything
else just below half a unit of 1, every addition that has a link of its own
drops its term: the error shows the chain's length.  It may not exceed that of
one product per thread and round on eight blocks an SM: 16 and 26 links for 18
and 34 vectors of the 1025 x 513 grid."""
import ctypes as C
import os

import numpy as np
import pytest

import mdz_build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("native") / "dots_probe.so")
    mdz_build._run([mdz_build._nvcc()] + mdz_build.NVCC_FLAGS + ["-shared", "-o", so,
                                                                os.path.join(HERE, "native", "dots_probe.cu")])
    return C.CDLL(so)


@pytest.mark.parametrize("nq,links", [(18, 16), (34, 26)])
def test_chain_of_fp32_sums(probe, nq, links):
    n = (1025 * 514 + 1026 * 513 + 1024 * 512 + 31) // 32 * 32
    rows = (nq + 7) // 8
    first = (152 * 4 + rows - 1) // rows * 256 * 4   # elements of the first round of loads
    b = np.full(n, 0.95 * 2.0 ** -24, np.float32)
    b[:first:4] = 1.0
    a = np.ones((nq, n), np.float32)
    out = np.zeros(nq)
    fp = C.POINTER(C.c_float)
    assert probe.probe_dots(nq, C.c_longlong(n), a.ctypes.data_as(fp), b.ctypes.data_as(fp),
                            out.ctypes.data_as(C.POINTER(C.c_double))) == 0
    exact = float(np.sum(b.astype(np.float64)))
    bound = (links - 1 + 5 + 1) * 2.0 ** -24
    assert np.all(np.abs(out - exact) <= bound * exact), (np.abs(out - exact).max() / exact * 2.0 ** 24, links + 5)
