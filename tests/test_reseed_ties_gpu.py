"""Nearest-marker search of the reseeding where its shortcut does not hold:
markers on a lattice around the new marker (equal and nearly equal distances:
the first in the reference's visiting order wins), crowded and empty quarter
cells, and a box narrower than the distances (the first visited marker is
copied).  Bit for bit against the oracle, which walks the cells in that order;
coordinates are multiples of 1/64 so that the squares are exact on both sides."""
import numpy as np
import pytest

import mdz
import oracle

pytestmark = pytest.mark.gpu

KEYS = ("vx", "vz", "sxxd", "szzd", "sxz", "strain", "strain_pl", "T", "cmul", "P")
ATTRS = (("sxxd", mdz.M_SXXD), ("szzd", mdz.M_SZZD), ("sxz", mdz.M_SXZ), ("strain_pl", mdz.M_STRAIN_PL),
         ("strain", mdz.M_STRAIN), ("T", mdz.M_T), ("cmul", mdz.M_CMUL), ("P", mdz.M_P))


def _case(kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "narrow":   # new markers lie up to 1.25 dz = 5 from a candidate, the box is 1 wide
        g = mdz.Grid(5, 9, 0.0, 1.0, 0.0, 32.0)
    else:
        g = mdz.Grid(17, 9, 0.0, 16.0, 0.0, 8.0)
    g.set_bc_pureshear(1.0)
    s = 8 if kind == "lattice" else 16
    X, Z = np.meshgrid(g.xg[0] + g.dx * (np.arange(s * g.ncx) + 0.5) / s, g.zg[0] + g.dz * (np.arange(s * g.ncz) + 0.5) / s)
    x, z = X.ravel(), Z.ravel()
    quarter = np.floor((x - g.xg[0]) / (g.dx / 2)).astype(int) * 1000 + np.floor((z - g.zg[0]) / (g.dz / 2)).astype(int)
    if kind == "lattice":       # whole quarter cells lost: their centres see rings of equals
        keep = rng.random(60000)[quarter] > 0.3
    elif kind == "narrow":      # only a marker or two per quarter cell, and some cells empty
        keep = (rng.random(len(x)) < 0.03) & (rng.random(60000)[quarter] > 0.3)
    else:                       # crowded: 64 a quarter cell next to empty ones
        keep = rng.random(60000)[quarter] > 0.5
    x, z = x[keep], z[keep]
    perm = rng.permutation(len(x))
    m = dict(x=x[perm], z=z[perm], phase=rng.integers(0, 3, len(x)).astype(np.int32))
    for k in KEYS:
        m[k] = rng.normal(size=len(x))
    return g, m


@pytest.mark.parametrize("kind", ["lattice", "crowded", "narrow"])
@pytest.mark.parametrize("seed", [1, 2])
def test_reseed_equal_distances(kind, seed):
    g, m = _case(kind, seed)
    cap = len(m["x"]) + 4 * g.ncx * g.ncz + 8
    o, o_added = oracle.reseed(g, m, cap, 16, 1)
    ctx = mdz.Context(g, 3, cap)
    ctx.set_markers(m["x"], m["z"], m["phase"])
    ctx.set_marker_velocity(m["vx"], m["vz"])
    for k, a in ATTRS:
        ctx.set_marker_attr(a, m[k])
    assert ctx.CountPartCell(1, 16, 1) == o_added and o_added > 0
    x, z, ph, vx, vz = ctx.get_markers()
    got = dict(x=x, z=z, phase=ph, vx=vx, vz=vz, **{k: ctx.get_marker_attr(a) for k, a in ATTRS})
    for k in got:
        assert np.array_equal(got[k], o[k]), (k, np.flatnonzero(got[k] != o[k])[:5])
    ctx.close()


def test_reseed_with_a_marker_outside_the_quarter_grid():
    """Such a marker has no position code: every search is the exact one."""
    g, m = _case("lattice", 3)
    m["x"][5], m["z"][9] = g.xg[-1] + 40 * g.dx, g.zg[0] - 1e9
    cap = len(m["x"]) + 4 * g.ncx * g.ncz + 8
    o, o_added = oracle.reseed(g, m, cap, 16, 1)
    ctx = mdz.Context(g, 3, cap)
    ctx.set_markers(m["x"], m["z"], m["phase"])
    ctx.set_marker_attr(mdz.M_T, m["T"])
    assert ctx.CountPartCell(1, 16, 1) == o_added and o_added > 0
    x, z, ph, _, _ = ctx.get_markers()
    assert np.array_equal(x, o["x"]) and np.array_equal(z, o["z"]) and np.array_equal(ph, o["phase"])
    assert np.array_equal(ctx.get_marker_attr(mdz.M_T), o["T"])
    ctx.close()
