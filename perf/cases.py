"""The work a program has this library do, as timed cases.

A case names a kind of call and its sizes.  The kinds, and what each stands
for in a run:

    step      one whole time step with the marker state owned by the host
              program, as in the reference's time loop: upload of the markers,
              mdz_time_step, download of the advected markers and of the grid
              velocity and pressure.  The lithosphere model (four phases,
              creep, elasticity, plasticity, gravity) in the plain FP64 form and in the
              FP32-refined form with the learned start, and the visco-elasto-
              plastic shear-band box (line search, softening).  The markers
              start near their yield stress and with a shear stress, as in the
              middle of a run; the lithosphere steps converge to 1e-10, so that a
              run's next step starts from stresses known to that.
    solve     one linear defect solve (FP64) of sinking inclusions: the linear problem
              a Picard iteration poses, on grids whose coarsest level is small
              and on grids whose cell counts stop halving early
    project   marker -> grid projection on device arrays: centroids or vertices,
              one- or nine-cell stencil, arithmetic / harmonic / geometric mean
    advect    RK4 advection of the resident markers through a convection cell,
              and the read-back of the markers
    rheology  the local visco-elasto-plastic solve of every node and phase with
              its tangent
    energy    one implicit energy step
    reseed    upload of thinned-out markers, one reseeding pass, read-back
    mlp       training of the learned local-rheology start from given weights

Inputs are seeded synthetic data with the value ranges of the package's own
configurations (mdz_setups).  Host arrays are page-locked, as a caller's
marker arrays would be.
"""
import ctypes as C
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "mdoodz6.0_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import mdz  # noqa: E402
import mdz_setups  # noqa: E402

ATTRS = (("sxxd", mdz.M_SXXD), ("szzd", mdz.M_SZZD), ("sxz", mdz.M_SXZ), ("strain_pl", mdz.M_STRAIN_PL),
         ("strain", mdz.M_STRAIN), ("T", mdz.M_T), ("cmul", mdz.M_CMUL), ("P", mdz.M_P))


# ---------------------------------------------------------------------------
def listed():
    return [
        # the benchmark model at its full size, FP32-refined form with the learned start
        dict(name="step_litho_1025x513_fp32", kind="step", model="lithosphere", Nx=1025, Nz=513, precision=32, learned=1,
             rel_tol=1e-10),
        # the same model at a resolution for parameter studies, plain FP64 form
        dict(name="step_litho_257x129_fp64", kind="step", model="lithosphere", Nx=257, Nz=129, precision=64, learned=0,
             rel_tol=1e-10),
        # the 401 x 401 visco-elasto-plastic box (cell counts halve four times, to 25 x 25)
        dict(name="step_shear_band_401_fp64", kind="step", model="shear_band", Nx=401, Nz=401, precision=64, learned=0,
             rel_tol=1e-8),
        # the linear-viscous inclusion benchmark's solve: the smallest system
        dict(name="solve_101", kind="solve", Nx=101, Nz=101, contrast=1e2, inclusions=1, rtol=1e-10),
        # 120 x 60 cells, a round-number resolution: halves twice, to 30 x 15
        dict(name="solve_121x61", kind="solve", Nx=121, Nz=61, contrast=1e1, inclusions=4, rtol=1e-10),
        # the time step's centroid projection at the benchmark's size: six fields and the phase fractions
        dict(name="project_centroids_1025x513", kind="project", Nx=1025, Nz=513, nm=4, fields=6, avg=0, phases=4,
             centroid=1, stencil=1),
        # nine-cell stencil on vertices, harmonic mean, five markers a side in an odd-sized grid
        dict(name="project_vertices9_302x151", kind="project", Nx=302, Nz=151, nm=5, fields=3, avg=1, phases=4,
             centroid=0, stencil=9),
        # 2.1 M markers through a convection cell
        dict(name="advect_513x257", kind="advect", Nx=513, Nz=257, nm=4),
        # local rheology of a layered lithosphere, mixed cells along the layer boundaries
        dict(name="rheology_513x257", kind="rheology", Nx=513, Nz=257, avg=0),
        # implicit heat diffusion, diffusion number 20 (a thin-cell grid's usual step)
        dict(name="energy_401", kind="energy", Nx=401, Nz=401, diffusion=20.0),
        # reseeding of a quarter-million markers, a tenth of them lost
        dict(name="reseed_201x101", kind="reseed", Nx=201, Nz=101, lost=0.1),
        # a short training of the learned start
        dict(name="mlp_train_50x65536", kind="mlp", steps=50, batch=65536),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "solve", "solve", "project", "project", "advect", "rheology", "energy",
                       "reseed", "mlp"])
    if kind == "step":
        # cell counts a multiple of 16, as any grid meant for multigrid
        if rng.random() < 0.67:
            nx = 16 * _log_int(rng, 6, 40)
            nz = 16 * max(4, int(nx / 16 * rng.uniform(0.4, 0.6)))
            form = rng.choice([(64, 0), (32, 1)])
            return dict(kind=kind, model="lithosphere", Nx=nx + 1, Nz=nz + 1, precision=form[0], learned=form[1],
                        rel_tol=1e-10)
        n = 16 * _log_int(rng, 5, 26)
        return dict(kind=kind, model="shear_band", Nx=n + 1, Nz=n + 1, precision=64, learned=0, rel_tol=1e-8)
    if kind == "solve":
        # any coarsest level up to 22 cells a side, doubled two to four times
        a, k = _log_int(rng, 5, 22), rng.choice([2, 3, 4])
        nx, nz = a << k, max(5, int(a * rng.uniform(0.5, 1.0))) << k
        return dict(kind=kind, Nx=nx + 1, Nz=nz + 1, contrast=10.0 ** rng.randint(0, 2), inclusions=rng.randint(1, 6),
                    rtol=1e-10)
    nx = _log_int(rng, 60, 900)
    nz = max(33, int(nx * rng.uniform(0.4, 0.6)))
    if kind == "project":
        return dict(kind=kind, Nx=nx, Nz=nz, nm=rng.choice([3, 4, 4, 5]), fields=rng.randint(1, 6),
                    avg=rng.choice([0, 0, 1, 2]), phases=rng.choice([0, 2, 4, 7]), centroid=rng.choice([0, 1]),
                    stencil=rng.choice([1, 1, 9]))
    if kind == "advect":
        return dict(kind=kind, Nx=nx, Nz=nz, nm=rng.choice([3, 4, 5]))
    if kind == "rheology":
        return dict(kind=kind, Nx=nx, Nz=nz, avg=rng.choice([0, 0, 2]))
    if kind == "energy":
        return dict(kind=kind, Nx=nx, Nz=nz, diffusion=round(10.0 ** rng.uniform(-1, 2), 3))
    if kind == "reseed":
        return dict(kind=kind, Nx=min(nx, 600), Nz=min(nz, 300), lost=round(rng.uniform(0.02, 0.2), 3))
    return dict(kind=kind, steps=rng.randint(10, 80), batch=_log_int(rng, 4096, 65536))


# ---------------------------------------------------------------------------
class Some:
    """A program's fields: the mdz_fields members it holds; the others stay NULL."""

    def __init__(self, **arrays):
        self.a = arrays

    def struct(self):
        s = mdz.FieldsStruct()
        for k, v in self.a.items():
            setattr(s, k, v.ctypes.data_as(C.POINTER(C.c_double)))
        return s


def _pinned(sizes, dtype=torch.float64):
    """Page-locked numpy arrays of the given lengths, in one block."""
    block = torch.zeros(sum(sizes), dtype=dtype, pin_memory=True).numpy()
    at = np.cumsum([0] + list(sizes))
    return [block[at[i]:at[i + 1]] for i in range(len(sizes))]


def _pin(a):
    b = torch.empty(a.size, dtype=torch.float64, pin_memory=True).numpy()
    b[:] = a.ravel()
    return b


class Markers:
    """Page-locked marker arrays of a fixed capacity, as a program allocates
    them once (Nb_part_max): n markers, the slots above are inactive."""

    def __init__(self, n, cap):
        d = _pinned([cap] * (4 + len(ATTRS)))
        self.n, self.x, self.z, self.vx, self.vz = n, d[0], d[1], d[2], d[3]
        self.attr = {a: v for (_, a), v in zip(ATTRS, d[4:])}
        self.phase = _pinned([cap], torch.int32)[0]
        self.phase[n:] = -1

    def upload(self, ctx):
        n = self.n
        ctx.set_marker_state(self.x[:n], self.z[:n], self.phase[:n], {a: v[:n] for a, v in self.attr.items()})

    def download(self, ctx, keys):
        ctx.get_marker_state((self.x, self.z, self.phase, self.vx, self.vz), {a: self.attr[a] for _, a in keys})
        self.n = ctx.n_markers
        out = dict(x=self.x, z=self.z, phase=self.phase, vx=self.vx, vz=self.vz, n=self.n)
        out.update({k: self.attr[a] for k, a in keys})
        return out


@functools.lru_cache(maxsize=2)
def _config(model, Nx, Nz, precision, learned, rel_tol):
    if model == "lithosphere":
        cfg = mdz_setups.config_lithosphere(Nx=Nx, Nz=Nz, precision=precision, learned=learned)
    else:
        cfg = mdz_setups.config_shear_band(N=Nx, precision=precision, learned=learned)
        cfg["model"].ispureshear_ale = 0   # every pass starts from the same box
    cfg["model"].rel_tol = rel_tol
    cfg["prestress"] = _prestress(cfg)
    return cfg


def _prestress(cfg):
    """A deviatoric normal stress near yield for each marker, by depth, and a shear stress."""
    m = cfg["markers"]
    if cfg["name"] == "lithosphere":
        sc = cfg["scales"]
        depth = -m["z"] * sc.L
        tau = 1e7 / sc.S * math.cos(math.pi / 6) + m["P"] * math.sin(math.pi / 6)
        s = 0.9 * np.minimum(tau, 6e7 / sc.S) * np.clip((25e3 - depth) / 10e3, 0.0, 1.0)
        return s, 0.2 * s * np.sin(6 * math.pi * m["x"] / (cfg["grid"].xmax - cfg["grid"].xmin))
    s = np.full(len(m["x"]), -0.97 * math.cos(math.pi / 6))
    return s, 0.02 * s * np.sin(6 * math.pi * m["x"]) * np.cos(math.pi * m["z"])


def _prepare_step(case, rng):
    cfg = _config(case["model"], case["Nx"], case["Nz"], case["precision"], case["learned"], case["rel_tol"])
    g, m = cfg["grid"], cfg["markers"]
    n = len(m["x"])
    cap = n + n // 8 + 4 * (g.Nx + g.Nz)
    ctx = mdz.Context(g, cfg["mat"].n_phases, cap)
    hin, out = Markers(n, cap), Markers(0, cap)
    hin.x[:n], hin.z[:n], hin.phase[:n] = m["x"], m["z"], m["phase"]
    for k, a in ATTRS:
        hin.attr[a][:n] = m[k]
    s, t = cfg["prestress"]
    hin.attr[mdz.M_SXXD][:n] = s
    hin.attr[mdz.M_SZZD][:n] = -s
    hin.attr[mdz.M_SXZ][:n] = t
    # cohesion varies from marker to marker, and some strain has been accumulated
    hin.attr[mdz.M_CMUL][:n] = 1.0 + 0.01 * rng.standard_normal(n)
    hin.attr[mdz.M_STRAIN_PL][:n] = 0.02 * rng.random(n)
    if case["learned"]:
        mdz_setups.train_guess(ctx, cfg)
    start = Some(**{k: _pin(np.asarray(cfg[k], np.float64)) for k in ("u", "v", "p")})
    uvp = [_pin(np.zeros(g.size(c))) for c in (-1, -2, 1)]
    return dict(kind="step", ctx=ctx, cfg=cfg, hin=hin, out=out, start=start, uvp=uvp)


def _run_step(s):
    ctx, cfg = s["ctx"], s["cfg"]
    s["hin"].upload(ctx)
    ctx.upload_fields(s["start"])
    rep = ctx.time_step(cfg["mat"], cfg["model"])
    out = s["out"].download(ctx, [k for k in ATTRS if k[0] not in ("T", "cmul")])
    dp = C.POINTER(C.c_double)
    ctx._check(ctx.L.mdz_get_velocity(ctx.h, *[a.ctypes.data_as(dp) for a in s["uvp"]]))
    out.update(u=s["uvp"][0], v=s["uvp"][1], p=s["uvp"][2], added=int(rep.markers_added), converged=int(rep.converged))
    return out


# ---------------------------------------------------------------------------
def _prepare_solve(case, rng):
    g = mdz.Grid(case["Nx"], case["Nz"], -0.5 * (case["Nx"] - 1) / (case["Nz"] - 1), 0.5 * (case["Nx"] - 1) / (case["Nz"] - 1),
                 -0.5, 0.5).set_bc_pureshear(1.0)
    blobs = [(rng.uniform(0.6 * g.xmin, 0.6 * g.xmax), rng.uniform(-0.3, 0.3), rng.uniform(0.08, 0.12),
              rng.uniform(0.5, 1.5)) for _ in range(case["inclusions"])]

    def inside(X, Z):
        w = np.zeros(X.shape)
        for x, z, r, b in blobs:
            w = np.maximum(w, b * (np.hypot(X - x, Z - z) < r))
        return w
    eta_n = np.where(inside(*np.meshgrid(g.xc, g.zc)) > 0, case["contrast"], 1.0).ravel()
    eta_s = np.where(inside(*np.meshgrid(g.xg, g.zg)) > 0, case["contrast"], 1.0).ravel()
    zero_n, zero_s = np.zeros_like(eta_n), np.zeros_like(eta_s)
    f = dict(eta_n=eta_n, eta_s=eta_s, D11_n=2 * eta_n, D22_n=2 * eta_n, D33_s=eta_s)
    for k in ("D12_n", "D13_n", "D14_n", "D21_n", "D23_n", "D24_n"):
        f[k] = zero_n
    for k in ("D31_s", "D32_s", "D34_s"):
        f[k] = zero_s
    # the right-hand side: the inclusions' weight on the Vz rows, a little on the Vx rows
    fv = (inside(*np.meshgrid(g.xvz, g.zg)).ravel() + 0.05 * np.sin(3 * np.repeat(g.zg, g.Nx + 1))) * g.dx * g.dz
    fu = 0.1 * np.cos(4 * np.repeat(g.zvx, g.Nx)) * g.dx * g.dz * rng.uniform(0.5, 1.5)
    fu, fv = fu * (g.BCu == -1), fv * (g.BCv == -1)
    return dict(kind="solve", ctx=mdz.Context(g, 1, 1), f=Some(**{k: _pin(v) for k, v in f.items()}), rtol=case["rtol"],
                F=(_pin(fu), _pin(fv), _pin(np.zeros(g.size(1)))))


def _run_solve(s):
    du, dv, dp, _, _ = s["ctx"].SolveStokesDefect(s["f"], 0, 64, s["rtol"], 2000, *s["F"])
    return dict(du=du, dv=dv, dp=dp)


# ---------------------------------------------------------------------------
def _seeded(case, rng, seed):
    """Markers some steps into a run: seeded cell by cell, then carried a few
    cells along by a smooth flow, one in a thousand lost."""
    g = mdz.Grid(case["Nx"], case["Nz"], 0.0, float(case["Nx"] - 1) / (case["Nz"] - 1), 0.0, 1.0).set_bc_pureshear(1.0)
    x, z = mdz_setups.seed_markers(g, case["nm"], case["nm"], 0.5, seed)
    w, h = g.xmax - g.xmin, g.zmax - g.zmin
    sx, sz = np.sin(math.pi * x / w), np.sin(math.pi * z / h)
    x, z = x + 2.5 * g.dx * sx * np.cos(math.pi * z / h), z - 2.5 * g.dz * sz * np.cos(math.pi * x / w)
    x, z = np.clip(x, g.xmin, g.xmax), np.clip(z, g.zmin, g.zmax)
    phase = np.minimum((z * max(1, case.get("phases", 4) or 4)).astype(np.int32), max(1, case.get("phases", 4) or 4) - 1)
    phase[rng.random(len(x)) < 1e-3] = -1
    return g, x, z, phase.astype(np.int32)


def _prepare_project(case, rng, seed):
    g, x, z, phase = _seeded(case, rng, seed)
    n = len(x)
    ctx = mdz.Context(g, max(1, case["phases"]), n)
    ctx.set_markers(x, z, phase)
    values = [np.exp(0.5 * rng.standard_normal(n)) for _ in range(case["fields"])]
    nn = g.size(case["centroid"])
    s = dict(kind="project", ctx=ctx, val=[torch.from_numpy(v).cuda() for v in values],
             out=[torch.zeros(nn, dtype=torch.float64, device="cuda") for _ in values],
             pp=torch.zeros((case["phases"], nn), dtype=torch.float64, device="cuda") if case["phases"] else None,
             avg=(C.c_int * len(values))(*[case["avg"]] * len(values)), centroid=case["centroid"], stencil=case["stencil"],
             host=(g, x, z, phase, values))
    pd = C.c_void_p * len(values)
    s["pv"], s["po"] = pd(*[t.data_ptr() for t in s["val"]]), pd(*[t.data_ptr() for t in s["out"]])
    return s


def _run_project(s):
    ctx = s["ctx"]
    ctx._check(ctx.L.mdz_dev_p2g(ctx.h, C.c_int(len(s["val"])), s["pv"], s["avg"], s["po"],
                                 C.c_void_p(s["pp"].data_ptr() if s["pp"] is not None else 0), C.c_int(s["centroid"]),
                                 C.c_int(s["stencil"]), None))
    return dict(fields=s["out"], phases=s["pp"])


def _exact_project(case, rng, seed):
    g, x, z, phase = _seeded(case, rng, seed)
    values = [np.exp(0.5 * rng.standard_normal(len(x))) for _ in range(case["fields"])]
    act = phase >= 0
    x, z, phase = x[act], z[act], phase[act]
    X, Z = (g.xc, g.zc) if case["centroid"] == 1 else (g.xg, g.zg)
    nx, nz, hw = len(X), len(Z), 1 if case["stencil"] == 9 else 0
    width = 1.5 if hw else 0.5
    ip = np.clip(np.ceil((x - X[0]) / g.dx + 0.5).astype(np.int64) - 1, 0, nx - 1)
    jp = np.clip(np.ceil((z - Z[0]) / g.dz + 0.5).astype(np.int64) - 1, 0, nz - 1)
    W, B = np.zeros(nx * nz), [np.zeros(nx * nz) for _ in values]
    P = np.zeros((case["phases"], nx * nz))
    tr = {0: lambda v: v, 1: lambda v: 1.0 / v, 2: np.log}[case["avg"]]
    back = {0: lambda v: v, 1: lambda v: 1.0 / v, 2: np.exp}[case["avg"]]
    tv = [tr(v[act]) for v in values]
    for dj in range(-hw, hw + 1):
        for di in range(-hw, hw + 1):
            ok = (ip + di >= 0) & (ip + di < nx) & (jp + dj >= 0) & (jp + dj < nz)
            i, j = ip[ok], jp[ok]
            w = (1 - np.abs(X[i] + di * g.dx - x[ok]) / (width * g.dx)) * (1 - np.abs(Z[j] + dj * g.dz - z[ok]) / (width * g.dz))
            node = (i + di) + (j + dj) * nx
            W += np.bincount(node, w, nx * nz)
            for b, v in zip(B, tv):
                b += np.bincount(node, w * v[ok], nx * nz)
            for p in range(case["phases"]):
                q = phase[ok] == p
                P[p] += np.bincount(node[q], w[q], nx * nz)
    have = np.abs(W) >= 1e-30
    Ws = np.where(have, W, 1.0)
    return dict(fields=[np.where(have, back(np.where(have, b / Ws, 1.0)), 0.0) for b in B],
                phases=P / Ws if case["phases"] else None)


# ---------------------------------------------------------------------------
def _cell_flow(g):
    """A convection cell that closes at the walls, on the staggered velocity nodes."""
    w, h = g.xmax - g.xmin, g.zmax - g.zmin
    u = np.sin(math.pi * g.xg / w)[None, :] * np.cos(math.pi * g.zvx / h)[:, None] * w
    v = -np.cos(math.pi * g.xvz / w)[None, :] * np.sin(math.pi * g.zg / h)[:, None] * h
    return u.ravel(), v.ravel(), 0.4 * g.dx / w


def _prepare_advect(case, rng, seed):
    g, x, z, phase = _seeded(case, rng, seed)
    ctx = mdz.Context(g, 4, len(x))
    ctx.set_markers(x, z, phase)
    u, v, dt = _cell_flow(g)
    n = len(x)
    out = _pinned([n] * 4)
    return dict(kind="advect", ctx=ctx, u=_pin(u), v=_pin(v), dt=dt,
                out=[out[0], out[1], _pinned([n], torch.int32)[0], out[2], out[3]])


def _run_advect(s):
    s["ctx"].RogerGuntherII(s["u"], s["v"], s["dt"])
    x, z, phase, vx, vz = s["ctx"].get_markers(s["out"])
    return dict(x=x, z=z, phase=phase, vx=vx, vz=vz)


def _exact_advect(case, rng, seed):
    g, x, z, phase = _seeded(case, rng, seed)
    u, v, dt = _cell_flow(g)

    def at(F, X, Z, x, z):
        nx = len(X)
        j = np.clip(np.ceil((x - X[0]) / g.dx).astype(np.int64) - 1, 0, nx - 2)
        i = np.clip(np.ceil((z - Z[0]) / g.dz).astype(np.int64) - 1, 0, len(Z) - 2)
        wx, wz = np.abs(x - X[j]) / g.dx, np.abs(z - Z[i]) / g.dz
        s = j + i * nx
        return (1 - wz) * ((1 - wx) * F[s] + wx * F[s + 1]) + wz * ((1 - wx) * F[s + nx] + wx * F[s + nx + 1])
    ph, xa, za = phase.copy(), x.copy(), z.copy()
    k = []
    for c in (0.5, 0.5, 1.0, None):
        on = ph != -1
        a, b = np.zeros_like(x), np.zeros_like(x)
        a[on], b[on] = at(u, g.xg, g.zvx, xa[on], za[on]), at(v, g.xvz, g.zg, xa[on], za[on])
        k.append((a, b))
        if c is None:
            break
        xa[on], za[on] = (x + c * dt * a)[on], (z + c * dt * b)[on]
        ph[(xa < g.xmin) | (xa > g.xmax) | (za < g.zmin) | (za > g.zmax)] = -1
    vx, vz = [(1.0 / 6.0) * (k[0][q] + 2 * k[1][q] + 2 * k[2][q] + k[3][q]) for q in (0, 1)]
    on = ph != -1
    xa[on], za[on] = (x + dt * vx)[on], (z + dt * vz)[on]
    ph[(xa < g.xmin) | (xa > g.xmax) | (za < g.zmin) | (za > g.zmax)] = -1
    vx[~on], vz[~on] = 0.0, 0.0
    return dict(x=xa, z=za, phase=ph, vx=vx, vz=vz)


# ---------------------------------------------------------------------------
RHEO_OUT = {"eta_n": 1, "eta_s": 0, "eta_phys_n": 1, "VE_n": 1, "sxxd": 1, "szzd": 1, "sxz": 0, "eII_el": 1, "eII_pl": 1,
            "eII_pwl": 1, "eII_lin": 1, "detadexx_n": 1, "detadezz_n": 1, "detadgxz_n": 1, "detadp_n": 1, "detadexx_s": 0,
            "detadezz_s": 0, "detadgxz_s": 0, "detadp_s": 0, "p_corr": 1, "Wdiss": 1}


def _prepare_rheology(case, rng):
    base = _config("lithosphere", 65, 33, 64, 0, 1e-8)   # the model's materials, scales and switches
    sc, mat = base["scales"], base["mat"]
    prm = mdz.RheoParams.from_buffer_copy(base["model"].rheo)
    prm.eta_avg = case["avg"]
    L = sc.L
    g = mdz.Grid(case["Nx"], case["Nz"], -500e3 / L, 500e3 / L, -400e3 / L, 0.0).set_bc_pureshear(1.0)
    eps = 0.01 / (365.25 * 24 * 3600) / 1000e3 / sc.E
    f = {}
    wave = rng.uniform(0, 2 * math.pi, 4)
    rho = (2700.0, 2900.0, 3300.0, 3300.0)
    for tail, X, Z in (("n", g.xc, g.zc), ("s", g.xg, g.zg)):
        depth = np.maximum(-Z[:, None] * L, 0.0) + 0.0 * X[None, :]
        shape, s = depth.shape, np.sin(2 * math.pi * X / (g.xmax - g.xmin) * 3 + wave[0])[None, :]
        below = [np.clip((depth - d - 4e3 * s) / (g.dz * L) + 0.5, 0.0, 1.0) for d in (20e3, 35e3, 120e3)]
        frac = np.stack([1 - below[0], below[0] * (1 - below[1]), below[1] * (1 - below[2]), below[2]])
        frac /= frac.sum(0)
        T = np.where(depth < 120e3, 273.15 + 1330.0 * depth / 120e3, 1603.15 + 0.3e-3 * (depth - 120e3))
        P = np.interp(depth, [0, 20e3, 35e3, 400e3], np.cumsum([0, 20e3 * rho[0], 15e3 * rho[1], 365e3 * rho[2]]) * 9.81) / sc.S
        e = eps * (1.0 + 0.5 * np.sin(2 * math.pi * 5 * X / (g.xmax - g.xmin) + wave[1])[None, :] + 0.05 * rng.standard_normal(shape))
        shear = 0.3 * eps * rng.standard_normal(shape)
        tau = 0.9 * np.minimum(1e7 / sc.S * math.cos(math.pi / 6) + 0.5 * P, 6e7 / sc.S) * np.clip((25e3 - depth) / 10e3, 0.0, 1.0)
        one = np.ones(shape)
        if tail == "n":
            f.update(exxd=e, ezzd=-e, exz_n=shear, sxxd0=tau, szzd0=-tau, sxz0_n=0.05 * tau, T=T, p=P * (1 + 0.01 * s), p0_n=P, d0_n=one)
        else:
            f.update(exxd_s=e, ezzd_s=-e, exz=shear, sxxd0_s=tau, szzd0_s=-tau, sxz0=0.05 * tau, p0_s=P)
        f.update({"phase_perc_" + tail: frac, "mu_" + tail: 3e10 / sc.S * one, "bet_" + tail: 1e-11 * sc.S * one,
                  "C_" + tail: 1e7 / sc.S * (1 + 0.01 * rng.standard_normal(shape)), "fric_" + tail: math.pi / 6 * one,
                  "dil_" + tail: 0.0 * one})
    out = {k: _pin(np.zeros(g.size(c))) for k, c in RHEO_OUT.items()}
    return dict(kind="rheology", ctx=mdz.Context(g, mat.n_phases, 1), mat=mat, prm=prm, out=out,
                f=Some(**{k: _pin(v) for k, v in f.items()}, **out))


def _run_rheology(s):
    s["ctx"].NonNewtonianViscosityGrid(s["mat"], s["prm"], s["f"])
    return s["out"]


# ---------------------------------------------------------------------------
def _energy_inputs(case, rng):
    g = mdz.Grid(case["Nx"], case["Nz"], 0.0, float(case["Nx"] - 1) / (case["Nz"] - 1), 0.0, 1.0).set_bc_pureshear(1.0)
    nx, nz = g.ncx, g.ncz
    Xc, Zc = np.meshgrid(g.xc, g.zc)
    f = dict(T=1.0 + 0.3 * np.sin(9 * Xc) * np.cos(7 * Zc) + 0.05 * rng.random(Xc.shape), rho_n=1.0 + 0.1 * rng.random(Xc.shape),
             Cv=0.8 + 0.4 * rng.random(Xc.shape), Qr=0.1 * rng.random(Xc.shape), Wdiss=0.2 * rng.random(Xc.shape),
             kx=np.exp(0.3 * rng.standard_normal(g.size(-1))), kz=np.exp(0.3 * rng.standard_normal(g.size(-2))))
    bc = dict(type=np.full(nx * nz, -1, np.int8), typS=np.ones(nx, np.int8), typN=np.ones(nx, np.int8),
              typW=np.zeros(nz, np.int8), typE=np.zeros(nz, np.int8), valS=1.2 + 0.1 * rng.random(nx),
              valN=0.5 + 0.1 * rng.random(nx), valW=np.zeros(nz), valE=np.zeros(nz))
    return g, f, bc, case["diffusion"] * min(g.dx, g.dz) ** 2


def _prepare_energy(case, rng):
    g, f, bc, dt = _energy_inputs(case, rng)
    T0 = f["T"].ravel().copy()
    f = {k: _pin(v) for k, v in f.items()}
    f["dT"] = _pin(np.zeros(g.size(1)))
    return dict(kind="energy", ctx=mdz.Context(g, 1, 1), f=Some(**f), bc=bc, dt=dt, T0=T0)


def _run_energy(s):
    np.copyto(s["f"].a["T"], s["T0"])   # the old temperature: the call writes the new one over it
    s["ctx"].EnergyDirectSolve(s["f"], s["bc"], s["dt"], 0.0, 1, 0)
    return dict(T=s["f"].a["T"], dT=s["f"].a["dT"])


def _exact_energy(case, rng):
    """The five-point system by conjugate gradients to rounding, with one refinement."""
    g, f, bc, dt = _energy_inputs(case, rng)
    nx, nz = g.ncx, g.ncz
    ixx, izz = 1.0 / g.dx / g.dx, 1.0 / g.dz / g.dz
    kx, kz = f["kx"].reshape(g.Nz + 1, g.Nx)[1:-1] * ixx, f["kz"].reshape(g.Nz, g.Nx + 1)[:, 1:-1] * izz
    c = f["rho_n"] * f["Cv"] / dt
    W, E, S, N = kx[:, :-1].copy(), kx[:, 1:].copy(), kz[:-1].copy(), kz[1:].copy()
    W[:, 0], E[:, -1] = 0.0, 0.0
    diag = c + W + E + S + N
    diag[0] += S[0]      # Dirichlet walls: twice the conductance to the wall
    diag[-1] += N[-1]
    b = c * f["T"] + f["Qr"] + f["Wdiss"]
    b[0] += 2 * S[0] * bc["valS"]
    b[-1] += 2 * N[-1] * bc["valN"]
    S, N = S.copy(), N.copy()
    S[0], N[-1] = 0.0, 0.0

    def apply(x):
        y = diag * x
        y[:, 1:] -= W[:, 1:] * x[:, :-1]
        y[:, :-1] -= E[:, :-1] * x[:, 1:]
        y[1:] -= S[1:] * x[:-1]
        y[:-1] -= N[:-1] * x[1:]
        return y
    x = f["T"].copy()
    for _ in range(2):
        r = b - apply(x)
        z = r / diag
        p, rz, stop = z.copy(), float((r * z).sum()), 1e-16 * float(np.linalg.norm(b))
        for _ in range(4000):
            if np.linalg.norm(r) <= stop:
                break
            q = apply(p)
            a = rz / float((p * q).sum())
            x += a * p
            r -= a * q
            z = r / diag
            new = float((r * z).sum())
            p = z + new / rz * p
            rz = new
    return dict(T=x.ravel(), dT=(x - f["T"]).ravel())


# ---------------------------------------------------------------------------
def _prepare_reseed(case, rng, seed):
    g, x, z, phase = _seeded(dict(case, nm=4), rng, seed)
    # clusters of markers lost: every k-th block of sixteen thinned to a random rest
    keep = rng.random(len(x)) >= case["lost"]
    x, z, phase = x[keep], z[keep], phase[keep]
    n, cap = len(x), 20 * g.ncx * g.ncz
    hin, out = Markers(n, cap), Markers(0, cap)
    hin.x[:n], hin.z[:n], hin.phase[:n] = x, z, phase
    for k, a in ATTRS:
        hin.attr[a][:n] = rng.standard_normal(n)
    grid = [rng.standard_normal(g.size(0 if q == 3 else 1)) for q in range(5)]
    return dict(kind="reseed", ctx=mdz.Context(g, 4, cap), hin=hin, out=out, grid=[_pin(a) for a in grid])


def _run_reseed(s):
    s["hin"].upload(s["ctx"])
    added = s["ctx"].CountPartCell(1, 16, 0, *s["grid"])
    got = s["out"].download(s["ctx"], ATTRS)
    got["added"] = added
    return got


# ---------------------------------------------------------------------------
def _prepare_mlp(case, rng):
    base = _config("lithosphere", 65, 33, 64, 0, 1e-8)
    ctx = mdz.Context(base["grid"], base["mat"].n_phases, 1)
    seed = int(rng.integers(1 << 30))
    ctx.mlp_init(seed)
    ctx.mlp_generate(base["mat"], base["model"].rheo, 1 << 20, seed, mdz_setups.LO_LITHO, mdz_setups.HI_LITHO)
    return dict(kind="mlp", ctx=ctx, w0=ctx.mlp_get_weights(), steps=case["steps"], batch=case["batch"])


def _run_mlp(s):
    ctx = s["ctx"]
    ctx.mlp_set_weights(s["w0"])
    loss = ctx.mlp_train(s["steps"], s["batch"], 2e-3)
    return dict(weights=ctx.mlp_get_weights(), loss=np.float32(loss))


# ---------------------------------------------------------------------------
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("project", "advect", "reseed"):
        return {"project": _prepare_project, "advect": _prepare_advect, "reseed": _prepare_reseed}[kind](case, rng, seed)
    return {"step": _prepare_step, "solve": _prepare_solve, "rheology": _prepare_rheology, "energy": _prepare_energy,
            "mlp": _prepare_mlp}[kind](case, rng)


def run(state):
    return {"step": _run_step, "solve": _run_solve, "project": _run_project, "advect": _run_advect, "rheology": _run_rheology,
            "energy": _run_energy, "reseed": _run_reseed, "mlp": _run_mlp}[state["kind"]](state)


def exact(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "project":
        return _exact_project(case, rng, seed)
    if case["kind"] == "advect":
        return _exact_advect(case, rng, seed)
    if case["kind"] == "energy":
        return _exact_energy(case, rng)
    return None   # implicit solves of a coupled system: no plain restatement


def work(case):
    """Bytes each input read once and each output written once, and a count of
    the arithmetic the path cannot do without."""
    if case["kind"] == "mlp":
        rows = case["steps"] * case["batch"]
        return {"bytes": 24.0 * rows, "flops": 27392.0 * rows}
    Nx, Nz = case["Nx"], case["Nz"]
    cells = (Nx - 1.0) * (Nz - 1.0)
    if case["kind"] == "step":
        n = 16.0 * cells   # markers: 8 attributes, x, z, phase in; 6 attributes, x, z, vx, vz, phase out
        return {"bytes": n * (84 + 84) + 6 * 8 * cells, "flops": 500.0 * n + 20000.0 * cells}
    if case["kind"] == "solve":
        return {"bytes": 8.0 * cells * 18, "flops": 20000.0 * cells}
    if case["kind"] == "project":
        n = cells * case["nm"] ** 2
        return {"bytes": n * (20 + 8 * case["fields"]) + 8 * cells * (case["fields"] + case["phases"]),
                "flops": n * case["stencil"] * (8 + 2 * case["fields"])}
    if case["kind"] == "advect":
        n = cells * case["nm"] ** 2
        return {"bytes": n * (20 + 36) + 16 * cells, "flops": 200.0 * n}
    if case["kind"] == "rheology":
        return {"bytes": 8 * cells * (33 + 8 + len(RHEO_OUT)), "flops": 2 * 600.0 * cells}
    if case["kind"] == "energy":
        return {"bytes": 8 * cells * 9, "flops": 40 * 20.0 * cells}
    n = 16 * cells * (1 - case["lost"])
    return {"bytes": n * (84 + 100) + 8 * 5 * cells, "flops": 50.0 * n}
