"""The energy step at the sizes where its one-launch solve splits differently:
fewer cells than one CTA holds, rows longer than a CTA's share of cells (the
halo then spans several CTAs), a last CTA that is nearly empty, shares that are
no multiple of the grid's row, every SM in use, and rows too long for shared
memory (one launch per step of the recurrence).  Against the oracle; the solve
stops at 1e-13 of the right-hand side and the rows' condition number is below
1e3, hence 1e-10 on T."""
import numpy as np
import pytest

import mdz
import oracle_thermal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx,Nz", [(3, 3), (5, 4), (17, 18), (33, 9), (1201, 4), (130, 259), (402, 401), (1026, 515),
                                   (9700, 4)])
def test_energy_step_sizes(Nx, Nz):
    from golden.make_golden import thermal_inputs
    g = mdz.Grid(Nx, Nz, 0.0, float(Nx - 1) / (Nz - 1), 0.0, 1.0).set_bc_pureshear(1.0)
    f, bc = thermal_inputs(np.random.default_rng(Nx), Nx - 1, Nz - 1, Nx, Nz)
    if Nx > 16 and Nz > 8:   # air, also across the ends of rows
        t = bc["type"].reshape(Nz - 1, Nx - 1)
        t[-3:, :5] = t[-3:, -7:] = 30
    dt = 5.0 * min(g.dx, g.dz) ** 2
    out = []
    ctx = mdz.Context(g, 1, 1)
    for _ in range(2):
        fl = mdz.GridFields(g, 1)
        for k, v in f.items():
            fl[k] = v
        out.append(ctx.EnergyDirectSolve(fl, bc, dt, -1.0, 1, 1) + (fl["T"].copy(), fl["dT"].copy()))
    ctx.close()
    T, dT = oracle_thermal.energy_step(Nx, Nz, g.dx, g.dz, f, bc, dt, -1.0, 1, 1)
    assert 0 < out[0][0] < 300 and out[0][1] <= 1e-13
    assert np.abs(out[0][2] - T).max() <= 1e-10 * np.abs(T).max()
    assert np.abs(out[0][3] - dT).max() <= 1e-8 * np.abs(dT).max()
    assert out[0][:2] == out[1][:2] and np.array_equal(out[0][2], out[1][2])   # fixed-order sums
