"""The tiled projection (4 rows of 32 nodes, four markers per node at a time) at
its edges: grids one node short of, at and past a tile, cells that are empty
or crowded, markers on cell and vertex lines and outside the box, air nodes,
both stencils, all means, one to twenty phases and up to eight fields at once.
Against the oracle; sums of positive terms in another order, 1e-12 as in the
other projection tests."""
import ctypes as C

import numpy as np
import pytest

import mdz
from oracle import Oracle

pytestmark = pytest.mark.gpu


def _uneven(Nx, Nz, nph, seed):
    g = mdz.Grid(Nx, Nz, -1.0, -1.0 + 2.0 * (Nx - 1) / (Nz - 1), 0.0, 2.0).set_bc_pureshear(1.0)
    rng = np.random.default_rng(seed)
    nc = g.ncx * g.ncz
    per = rng.choice([0, 1, 3, 4, 5, 9, 16, 41], nc, p=[0.1, 0.1, 0.1, 0.2, 0.1, 0.15, 0.2, 0.05])
    c = np.repeat(np.arange(nc), per)
    x = g.xg[c % g.ncx] + g.dx * rng.random(len(c))
    z = g.zg[c // g.ncx] + g.dz * rng.random(len(c))
    on = np.array([(a, b) for a in (g.xg[0], g.xg[-1], g.xc[0], g.xg[1]) for b in (g.zg[0], g.zg[-1], g.zc[-1], g.zg[1])])
    x = np.concatenate([x, on[:, 0], [g.xg[0] - 0.2 * g.dx, g.xg[-1] + 0.2 * g.dx]])
    z = np.concatenate([z, on[:, 1], [g.zg[-1] + 0.2 * g.dz, g.zg[0] - 0.2 * g.dz]])
    ph = rng.integers(0, nph, len(x)).astype(np.int32)
    ph[rng.random(len(x)) < 0.05] = -1
    perm = rng.permutation(len(x))
    return g, x[perm], z[perm], ph[perm]


def _defined(g, x, z, ph, centroid, stencil):
    """Nodes with no marker, or with a weight that is not the rounding of zero: a
    marker half-way between two lines weighs 1 - 1, and a node that holds only
    such markers takes their mean or keeps its value by the last bit of that."""
    X = {1: g.xc, 0: g.xg, -1: g.xg, -2: g.xvz}[centroid]
    Z = {1: g.zc, 0: g.zg, -1: g.zvx, -2: g.zg}[centroid]
    x, z = x[ph >= 0], z[ph >= 0]
    nx, nz, h = len(X), len(Z), int(stencil == 9)
    ip = np.clip(np.ceil((x - X[0]) / g.dx + 0.5).astype(int) - 1, 0, nx - 1)
    jp = np.clip(np.ceil((z - Z[0]) / g.dz + 0.5).astype(int) - 1, 0, nz - 1)
    W, n = np.zeros(nx * nz), np.zeros(nx * nz, int)
    for dj in range(-h, h + 1):
        for di in range(-h, h + 1):
            ok = (ip + di >= 0) & (ip + di < nx) & (jp + dj >= 0) & (jp + dj < nz)
            w = ((1 - np.abs(X[ip] + di * g.dx - x) / (g.dx * (h + 0.5)))
                 * (1 - np.abs(Z[jp] + dj * g.dz - z) / (g.dz * (h + 0.5))))[ok]
            at = ((ip + di) + (jp + dj) * nx)[ok]
            np.add.at(W, at, w)
            np.add.at(n, at, 1)
    return (n == 0) | (np.abs(W) > 1e-9)


@pytest.mark.parametrize("Nx,Nz,nph", [(3, 3, 1), (3, 5, 2), (32, 4, 4), (33, 5, 5), (34, 6, 20), (65, 9, 4), (31, 66, 3)])
def test_p2g_at_tile_edges(Nx, Nz, nph):
    g, x, z, ph = _uneven(Nx, Nz, nph, Nx + Nz)
    rng = np.random.default_rng(2)
    vals = np.exp(rng.normal(size=len(x)))
    ctx = mdz.Context(g, nph, len(x))
    ctx.set_markers(x, z, ph)
    o = Oracle(g, nph)
    o.set_markers(x, z, ph)
    for centroid in (1, 0, -1, -2):
        tags = g.tags(centroid).copy()
        tags[::7] = 30
        for stencil in (1, 9):
            ok = _defined(g, x, z, ph, centroid, stencil)
            for avg in (0, 1, 2):
                init = np.full(g.size(centroid), 3.0)
                for flag, v in ((1, vals), (0, np.arange(1.0, nph + 1))):
                    got = ctx.P2Mastah(v, init, tags, flag, avg, 0, centroid, stencil)
                    want = o.P2Mastah(v, init, tags, flag, avg, 0, centroid, stencil)
                    np.testing.assert_allclose(got[ok], want[ok], rtol=1e-12, atol=1e-15 if avg == 2 else 0,
                                               err_msg="c%d s%d a%d f%d" % (centroid, stencil, avg, flag))
            if centroid >= 0:
                got = ctx.P2Mastah(np.ones(nph), None, tags, 0, 0, 1, centroid, stencil)
                want = o.P2Mastah(np.ones(nph), None, tags, 0, 0, 1, centroid, stencil)
                np.testing.assert_allclose(got.reshape(nph, -1)[:, ok], want.reshape(nph, -1)[:, ok], rtol=1e-12, atol=1e-15)
    c, v, pc, pv = ctx.count_markers()
    oc, ov, opc, opv = o.count_markers()
    assert np.array_equal(c, oc) and np.array_equal(v, ov) and np.array_equal(pc, opc) and np.array_equal(pv, opv)
    ctx.close()


@pytest.mark.parametrize("nf", [1, 2, 5, 8])
@pytest.mark.parametrize("stencil", [1, 9])
def test_fields_together_as_one_by_one(nf, stencil):
    import torch
    g, x, z, ph = _uneven(70, 37, 4, 5)
    rng = np.random.default_rng(3)
    vals = [np.exp(rng.normal(size=len(x))) for _ in range(nf)]
    ctx = mdz.Context(g, 4, len(x))
    ctx.set_markers(x, z, ph)
    for centroid in (1, 0):
        avg = [f % 3 for f in range(nf)]
        d = [torch.from_numpy(v).cuda() for v in vals]
        out = [torch.zeros(g.size(centroid), dtype=torch.float64, device="cuda") for _ in vals]
        P = C.c_void_p * nf
        torch.cuda.synchronize()
        ctx._check(ctx.L.mdz_dev_p2g(ctx.h, C.c_int(nf), P(*[t.data_ptr() for t in d]), (C.c_int * nf)(*avg),
                                     P(*[t.data_ptr() for t in out]), None, C.c_int(centroid), C.c_int(stencil), None))
        for f in range(nf):
            one = ctx.P2Mastah(vals[f], np.zeros(g.size(centroid)), g.tags(centroid), 1, avg[f], 0, centroid, stencil)
            assert np.array_equal(out[f].cpu().numpy(), one)
    ctx.close()
