"""The marker kernels read the index ceil(d/h + add) - 1 from the mantissa of
fma(d, 1/h, add + 1.5 2^32) (line_index in csrc/mdz_internal.cuh) and fall back
to the quotient within two units of 2^-20 of an integer.  The rule on the CPU,
with the fused product in extended precision, against the plain division, on
random positions and on positions on and around every line; quarter-cell
indices likewise against the reference's quotient, product and sum."""
import numpy as np
import pytest

from test_index_fastpath import lines

MAGIC = 6442450944.0


def line_index(d, ih, add):
    t = (np.longdouble(d) * np.longdouble(ih) + np.longdouble(add + MAGIC)).astype(np.float64)
    b = t.view(np.uint64)
    hi, lo = (b >> np.uint64(32)).astype(np.uint32), (b & np.uint64(0xffffffff)).astype(np.uint32)
    i = (((hi << np.uint32(12)) | (lo >> np.uint32(20))) ^ np.uint32(0x80000000)).view(np.int32)
    sure = (hi >> np.uint32(20) == 0x41f) & ((lo & np.uint32(0xfffff)) - np.uint32(2) <= 0xffffc)
    return i, sure


def positions(n, x0, x1, h):
    rng = np.random.default_rng(n)
    L = lines(x0, h, n)
    pts = [rng.uniform(x0 - 2 * h, x1 + 2 * h, 200000), L, L + h / 2, L + h / 4]
    for e in np.ldexp(h, -np.arange(15, 50)):
        pts += [L + e, L - e, L + h / 2 + e, L + h / 2 - e]
    return np.concatenate(pts), L


@pytest.mark.parametrize("n,x0,x1", [(3, 0.0, 1.0), (33, -7.3, 11.9), (513, -0.5, 0.0), (1025, -1.0, 1.0),
                                     (65535, -1e5, 3e5)])
def test_line_index_matches_division(n, x0, x1):
    h = (x1 - x0) / (n - 1)
    x, L = positions(n, x0, x1, h)
    for add in (0.0, 0.5):
        for X0 in (x0, L[0] + h / 2, L[0] - h / 2):
            d = x - X0
            i, sure = line_index(d, 1.0 / h, add)
            np.testing.assert_array_equal(i[sure], (np.ceil(d / h + add) - 1)[sure].astype(np.int32))
    d = x - (L[0] - h / 2 - h / 4)   # quarter cells: ceil(((x - q0) / h) 2 + 0.5) - 1
    i, sure = line_index(d, 2.0 / h, 0.5)
    np.testing.assert_array_equal(i[sure], (np.ceil(d / h * 2.0 + 0.5) - 1)[sure].astype(np.int32))


@pytest.mark.parametrize("n,x0,x1", [(3, 0.0, 1.0), (33, -7.3, 11.9), (513, 1e6, 1e6 + 0.5), (1025, -1.0, 1.0)])
def test_ghosted_index_by_integer_sum(n, x0, x1):
    """line_indices (csrc/mdz_internal.cuh): the index on the lines half a cell
    below from the same mantissa plus the rounded distance of the first lines."""
    h = (x1 - x0) / (n - 1)
    x, L = positions(n, x0, x1, h)
    xh0 = x0 - h / 2
    off = np.int64(np.rint((x0 - xh0) * (1.0 / h) * 1048576.0))
    t = (np.longdouble(x - x0) * np.longdouble(1.0 / h) + np.longdouble(MAGIC)).astype(np.float64)
    a = t.view(np.int64)
    b = a + off
    sure = ((a & 0xfffff) - 3 >= 0) & ((a & 0xfffff) - 3 <= 0xffffa) & ((b & 0xfffff) - 3 >= 0) & ((b & 0xfffff) - 3 <= 0xffffa)
    assert sure.any() and ((a >> 52) == 0x41f).all()
    for m, X0 in ((a, x0), (b, xh0)):
        i = (((m >> 20) & 0xffffffff).astype(np.uint32) ^ np.uint32(0x80000000)).view(np.int32)
        np.testing.assert_array_equal(i[sure], (np.ceil((x - X0) / h) - 1)[sure].astype(np.int32))


def test_line_index_leaves_the_rest_to_the_quotient():
    d = np.array([np.nan, np.inf, -np.inf, 1e300, -3e9, 2.2e9, 0.0, 1.0, 1.0 + 2.0 ** -20])
    assert not line_index(d, 1.0, 0.0)[1].any()


@pytest.mark.gpu
def test_advection_box_test():
    """Positions on the walls stay, the next number beyond leaves; -0 is 0 and a NaN never leaves."""
    import mdz
    g = mdz.Grid(9, 9, 0.0, 1.0, -2.0, 0.0).set_bc_pureshear(1.0)
    tiny = np.float64(5e-324)
    x = np.array([0.0, -0.0, 1.0, -tiny, np.nextafter(1.0, 2.0), tiny, 0.5, 0.5, 0.5, 0.5, 0.5, 0.5, np.nan, -np.inf])
    z = np.array([-1.0, -1.0, -1.0, -1.0, -1.0, -1.0, 0.0, -0.0, tiny, -2.0, np.nextafter(-2.0, -3.0), -tiny, -1.0, -1.0])
    out = np.array([0, 0, 0, 1, 1, 0, 0, 0, 1, 0, 1, 0, 0, 0], bool)   # at -inf the weights give inf 0 = NaN first
    ctx = mdz.Context(g, 1, len(x))
    ctx.set_markers(x, z, np.zeros(len(x), np.int32))
    ctx.RogerGuntherII(np.zeros(9 * 10), np.zeros(10 * 9), 0.1)
    got = ctx.get_markers()
    np.testing.assert_array_equal(got[2], np.where(out, -1, 0))
    ctx.close()
