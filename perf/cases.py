"""Performance cases: the work that a two-phase flow program has this package do.

A projection step transports and reinitializes the interface field, predicts the
velocity, solves a variable-density pressure-Poisson system and corrects the
velocity; nearly all of that is compact (CCD) line solves and Krylov
iterations.  The cases are those parts, each through the class a program
constructs once and calls every step, from the 64^2 quick-start grid (where a
call is launches and latency) to 256^3 (where it is memory traffic).

Fields are node-centred on the unit box, ``N + 1`` nodes per axis.  ``exact``
restates every path in FP64 torch: the CCD derivatives as dense matrices, the
pressure solve as conjugate gradients to round-off.
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import torch

import twophaseflow_b200 as tpf
from twophaseflow_b200.learned import PPESolverLearned

REYNOLDS, FROUDE, WEBER = 100.0, 1.0, 10.0


# ---- the cases --------------------------------------------------------------------------------
def listed():
    return [
        # one derivative pair per axis on the quick-start grid: the smallest call
        {"name": "ccd_2d_64", "kind": "ccd", "n0": 64, "n1": 64, "n2": 0, "bc": "wall", "dtype": "f64"},
        # the 2-D operator benchmark
        {"name": "ccd_2d_1024", "kind": "ccd", "n0": 1024, "n1": 1024, "n2": 0, "bc": "wall", "dtype": "f64"},
        # the 3-D operator benchmark, the largest field
        {"name": "ccd_3d_256", "kind": "ccd", "n0": 256, "n1": 256, "n2": 256, "bc": "wall", "dtype": "f64"},
        # single precision in a periodic box of unequal, odd sides
        {"name": "ccd_3d_f32_periodic", "kind": "ccd", "n0": 191, "n1": 160, "n2": 225, "bc": "periodic",
         "dtype": "f32"},
        # interface transport (RK3, mass-corrected) and reinitialization of the 192^3 rising-bubble step
        {"name": "levelset_3d_192", "kind": "levelset", "n0": 192, "n1": 192, "n2": 192, "bc": "wall"},
        # momentum predictor of a 3-D step: convection, gravity, surface tension, Picard Crank-Nicolson viscosity
        {"name": "predictor_3d", "kind": "predictor", "n0": 128, "n1": 96, "n2": 161, "convection": "ccd",
         "rho_g": 1e-3},
        # the 2-D work around a pressure solve: curvature, Rhie-Chow right-hand side, velocity correction
        {"name": "projection_2d_1024", "kind": "projection", "n0": 1024, "n1": 1024, "n2": 0, "rho_g": 1e-3},
        # the headline pressure solve: plain FP64 PCG to 1e-8, 12 droplets, density ratio 1000
        {"name": "ppe_cg_512", "kind": "cg", "n0": 512, "n1": 512, "n2": 0, "tol": 1e-8, "rho_g": 1e-3},
        # the 3-D pressure solve, to the tighter tolerance that parity runs use
        {"name": "ppe_cg_3d_128", "kind": "cg", "n0": 128, "n1": 128, "n2": 128, "tol": 1e-10, "rho_g": 1e-3},
        # the quick-start pressure solve: GMRES(80), exact line preconditioner, density ratio 10
        {"name": "ppe_gmres_64", "kind": "gmres", "n0": 64, "n1": 64, "n2": 0, "tol": 1e-10, "rho_g": 0.1},
        # the learned solve of the same system: flexible GMRES(60) with the shipped network
        {"name": "ppe_learned_512", "kind": "learned", "n0": 512, "n1": 512, "n2": 0, "tol": 1e-10, "rho_g": 1e-3},
        # a parameter sweep: many independent small pressure systems in one call
        {"name": "ppe_batch_32", "kind": "batch", "count": 32, "n0": 48, "n1": 96, "tol": 1e-10, "rho_g": 1e-3},
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of lo..hi, odd and even alike."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo2, hi2, lo3, hi3):
    """Sides of a 2-D or 3-D grid: unequal, within a factor of 1.5 of one another."""
    two = rng.random() < 0.5
    lo, hi = (lo2, hi2) if two else (lo3, hi3)
    n = _log_int(rng, lo, hi)
    side = [max(lo, min(hi, int(n * rng.uniform(0.8, 1.2)))) for _ in range(3)]
    return {"n0": side[0], "n1": side[1], "n2": 0 if two else side[2]}


def draw(rng):
    kind = rng.choice(["ccd", "ccd", "ccd", "levelset", "predictor", "projection", "cg", "cg", "gmres", "learned",
                       "batch"])
    if kind == "ccd":
        return {"kind": kind, **_box(rng, 33, 1024, 24, 256), "bc": rng.choice(["wall", "periodic"]),
                "dtype": rng.choice(["f64", "f64", "f32"])}
    if kind == "levelset":
        return {"kind": kind, **_box(rng, 64, 1024, 24, 192), "bc": rng.choice(["wall", "wall", "periodic"])}
    if kind == "predictor":
        return {"kind": kind, **_box(rng, 64, 768, 24, 144), "convection": rng.choice(["ccd", "uccd6"]),
                "rho_g": rng.choice([1e-3, 1e-2, 1e-1])}
    if kind == "projection":
        return {"kind": kind, **_box(rng, 64, 1024, 24, 160), "rho_g": rng.choice([1e-3, 1e-2, 1e-1])}
    if kind == "cg":
        return {"kind": kind, **_box(rng, 48, 512, 24, 128), "tol": 1e-10, "rho_g": rng.choice([1e-3, 1e-2, 1e-1])}
    if kind == "gmres":
        n = _log_int(rng, 32, 128)
        return {"kind": kind, "n0": n, "n1": max(32, int(n * rng.uniform(0.8, 1.2))), "n2": 0, "tol": 1e-10,
                "rho_g": 0.1}
    if kind == "learned":
        n = rng.randint(400, 512)
        return {"kind": kind, "n0": n, "n1": rng.randint(400, 512), "n2": 0, "tol": 1e-10,
                "rho_g": rng.choice([1e-3, 1e-2])}
    lo = rng.randint(32, 64)
    return {"kind": kind, "count": rng.randint(6, 32), "n0": lo, "n1": lo + rng.randint(0, 32), "tol": 1e-10,
            "rho_g": rng.choice([1e-3, 1e-2])}


def _cells(case):
    return tuple(case[k] for k in ("n0", "n1", "n2") if case.get(k))


def _points(case):
    n = 1
    for c in _cells(case):
        n *= c + 1
    return n


def _batch_grids(case):
    """Sizes of a batch's systems: spread over n0..n1 cells per axis."""
    c, lo, hi = case["count"], case["n0"], case["n1"]
    at = [lo + (hi - lo) * k // max(1, c - 1) for k in range(c)]
    return [(at[k], at[(7 * k + 3) % c]) for k in range(c)]


# ---- seeded inputs ----------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed):
    return torch.Generator(device="cpu").manual_seed(int(seed))


def _axes(N):
    return [torch.linspace(0.0, 1.0, n + 1, dtype=torch.float64, device=_dev()) for n in N]


def _along(v, axis, ndim):
    shape = [1] * ndim
    shape[axis] = -1
    return v.reshape(shape)


def _sync_images(f, bc="periodic"):
    """Node N of every axis takes node 0's value, as a periodic field stores it."""
    if bc == "periodic":
        for ax in range(f.dim()):
            f.select(ax, -1).copy_(f.select(ax, 0))
    return f


def _modes(N, g, count=16, kmax=24):
    """A smooth box-periodic field: sum of seeded cosine products, amplitude 1/|k|^2."""
    nd, ax = len(N), _axes(N)
    k = torch.randint(1, kmax + 1, (count, nd), generator=g).double()
    amp = torch.randn(count, generator=g, dtype=torch.float64) / (k * k).sum(1)
    ph = 2 * math.pi * torch.rand(count, nd, generator=g, dtype=torch.float64)
    f = torch.zeros([n + 1 for n in N], dtype=torch.float64, device=_dev())
    for m in range(count):
        t = float(amp[m])
        for d in range(nd):
            t = t * _along(torch.cos(2 * math.pi * float(k[m, d]) * ax[d] + float(ph[m, d])), d, nd)
        f += t
    return _sync_images(f)


def _velocity(N, g, bc="wall"):
    """Seeded velocity of order one: no flow through walls, or box-periodic."""
    nd, ax = len(N), _axes(N)
    out = []
    for d in range(nd):
        u = torch.zeros([n + 1 for n in N], dtype=torch.float64, device=_dev())
        for _ in range(4):
            k = torch.randint(1, 5, (nd,), generator=g).double()
            t = float(torch.randn(1, generator=g, dtype=torch.float64)) / float(k.sum())
            for e in range(nd):
                w = (1.0 if bc == "wall" else 2.0) * math.pi * float(k[e])
                t = t * _along(torch.sin(w * ax[e]) if e == d else torch.cos(w * ax[e]), e, nd)
            u += t
        out.append(_sync_images(u, bc))
    return out


def _droplets(N, g, count=12):
    """psi = 1 in ``count`` seeded, separate droplets, 0 in the gas, interface 1.5 h wide."""
    nd, ax = len(N), _axes(N)
    placed = []
    while len(placed) < count:
        v = torch.rand(nd + 1, generator=g, dtype=torch.float64).tolist()
        r = 0.02 + 0.06 * v[nd]
        c = [r + 0.02 + x * (1.0 - 2.0 * (r + 0.02)) for x in v[:nd]]
        if all(math.dist(c, c2) >= r + r2 + 0.02 for c2, r2 in placed):
            placed.append((c, r))
    phi = torch.full([n + 1 for n in N], math.inf, dtype=torch.float64, device=_dev())
    for c, r in placed:
        d2 = sum(_along((ax[d] - c[d]) ** 2, d, nd) for d in range(nd))
        phi = torch.minimum(phi, torch.sqrt(d2) - r)
    return torch.sigmoid(-phi * (max(N) / 1.5)).contiguous()


def _bubble(N, g):
    """psi = 0 in one gas bubble near the centre, 1 in the liquid."""
    nd, ax = len(N), _axes(N)
    v = torch.rand(nd + 1, generator=g, dtype=torch.float64).tolist()
    d2 = sum(_along((ax[d] - 0.45 - 0.1 * v[d]) ** 2, d, nd) for d in range(nd))
    return torch.sigmoid((torch.sqrt(d2) - 0.2 - 0.05 * v[nd]) * (max(N) / 1.5)).contiguous()


def _divergence(N, g):
    """A pressure right-hand side: divergence of a smooth seeded velocity."""
    nd, ax = len(N), _axes(N)
    f = torch.zeros([n + 1 for n in N], dtype=torch.float64, device=_dev())
    for _ in range(8):
        k = torch.randint(1, 9, (nd,), generator=g).double()
        ph = 2 * math.pi * torch.rand(nd, generator=g, dtype=torch.float64)
        amp = torch.randn(nd, generator=g, dtype=torch.float64)
        t = float((amp * k).sum()) * math.pi
        for d in range(nd):
            t = t * _along(torch.cos(math.pi * float(k[d]) * ax[d] + float(ph[d])), d, nd)
        f += t
    return f


def _inputs(case, seed):
    g, kind, N = _gen(seed), case["kind"], _cells(case)
    if kind == "ccd":
        f = _modes(N, g, count=24 if len(N) == 2 else 12, kmax=max(2, min(64, min(N) // 6)))
        return {"f": f.to(torch.float32 if case["dtype"] == "f32" else torch.float64)}
    if kind == "levelset":
        vel = _velocity(N, g, case["bc"])
        top = sum(float(v.abs().max()) for v in vel)
        return {"psi": _sync_images(_droplets(N, g), case["bc"]), "vel": vel, "dt": 0.3 / max(N) / top}
    if kind in ("predictor", "projection"):
        psi = _bubble(N, g)
        s = {"psi": psi, "rho": case["rho_g"] + (1.0 - case["rho_g"]) * psi, "vel": _velocity(N, g),
             "p": _modes(N, g, count=8, kmax=6)}
        s["dt"] = 0.1 / max(N) ** 1.5
        if kind == "predictor":
            s["mu"] = 0.01 + 0.99 * psi
            s["kappa"] = 8.0 * 4.0 * psi * (1.0 - psi) * (1.0 + _modes(N, g, count=4, kmax=4))
        return s
    if kind == "batch":
        return {"systems": [_system(n, g, case) for n in _batch_grids(case)]}
    return _system(N, g, case)


def _system(N, g, case):
    psi = _bubble(N, g) if case["kind"] == "gmres" else _droplets(N, g)
    return {"rhs": _divergence(N, g), "rho": case["rho_g"] + (1.0 - case["rho_g"]) * psi}


# ---- what a program keeps, and one pass -------------------------------------------------------
def _ppe_config(case, method):
    return SimpleNamespace(pseudo_tol=case["tol"], pseudo_maxiter=20000 if method == "cg" else 500,
                           ppe_iteration_method=method,
                           ppe_preconditioner="jacobi" if method == "cg" else "line_pcr")


def prepare(case, seed):
    s = _inputs(case, seed)
    kind, N = case["kind"], _cells(case)
    s["kind"] = kind
    if kind == "batch":
        s["solvers"] = [tpf.PPESolverFVMMatrixFree(None, _ppe_config(case, "cg"), tpf.UniformGrid(n))
                        for n in _batch_grids(case)]
        return s
    grid = tpf.UniformGrid(N)
    if kind in ("cg", "gmres"):
        s["solver"] = tpf.PPESolverFVMMatrixFree(None, _ppe_config(case, kind), grid)
        return s
    if kind == "learned":
        s["solver"] = PPESolverLearned(None, _ppe_config(case, "cg"), grid)
        return s
    ccd = tpf.CCDSolver(grid, None, bc_type=case.get("bc", "wall"),
                        dtype=torch.float32 if case.get("dtype") == "f32" else torch.float64)
    s["ccd"] = ccd
    if kind == "levelset":
        fccd = tpf.FCCDSolver(grid, None, bc_type=case["bc"], ccd_solver=ccd)
        s["transport"] = tpf.FCCDLevelSetAdvection(None, grid, fccd, mass_correction=True)
        s["reinit"] = tpf.SplitReinitializer(None, grid, ccd, 1.5 / max(N),
                                             bc="periodic" if case["bc"] == "periodic" else "neumann")
    elif kind == "predictor":
        cfg = SimpleNamespace(grid=SimpleNamespace(ndim=len(N)),
                              fluid=SimpleNamespace(Re=REYNOLDS, Fr=FROUDE, We=WEBER),
                              numerics=SimpleNamespace(cn_viscous=True, cn_mode="picard"))
        conv = tpf.UCCD6ConvectionTerm(None, grid, ccd) if case["convection"] == "uccd6" else None
        s["predictor"] = tpf.Predictor(None, cfg, ccd, convection=conv)
    elif kind == "projection":
        s["curvature"] = tpf.CurvatureCalculatorPsi(None, ccd)
        s["rhie_chow"] = tpf.RhieChowInterpolator(None, grid, ccd, bc_type="wall")
        s["corrector"] = tpf.VelocityCorrector(None, grid, ccd)
    return s


def run(s):
    kind = s["kind"]
    if kind == "ccd":
        return [s["ccd"].differentiate(s["f"], ax) for ax in range(s["f"].dim())]
    if kind == "levelset":
        moved = s["transport"].advance(s["psi"], s["vel"], s["dt"])
        return {"moved": moved, "sharp": s["reinit"].reinitialize(moved)}
    if kind == "predictor":
        st = tpf.FlowState(velocity=s["vel"], psi=s["psi"], rho=s["rho"], mu=s["mu"], kappa=s["kappa"],
                           pressure=s["p"])
        return s["predictor"].compute(st, s["dt"])
    if kind == "projection":
        return {"kappa": s["curvature"].compute(s["psi"]),
                "div": s["rhie_chow"].face_velocity_divergence(s["vel"], s["p"], s["rho"], s["dt"]),
                "vel": s["corrector"].correct(s["vel"], s["p"], s["rho"], s["dt"])}
    if kind == "batch":
        return tpf.solve_batched(s["solvers"], [y["rhs"] for y in s["systems"]], [y["rho"] for y in s["systems"]])
    return s["solver"].solve(s["rhs"], s["rho"])


def work(case):
    """Every input field read once, every output written once; for the solves that is what the whole
    solve cannot do without, however many iterations the method takes."""
    kind, nd = case["kind"], len(_cells(case))
    if kind == "ccd":
        es = 4 if case["dtype"] == "f32" else 8
        return {"bytes": 3.0 * nd * es * _points(case), "flops": 30.0 * nd * _points(case)}
    if kind == "batch":
        n = sum((a + 1) * (b + 1) for a, b in _batch_grids(case))
        return {"bytes": 24.0 * n, "flops": 20.0 * n}
    n = _points(case)
    fields, flops = {
        "levelset": (nd + 3, 3 * nd * 30 + 4 * nd * 70),           # psi, velocity in; two psi out
        "predictor": (2 * nd + 5, (3 * nd * nd + 2 * nd) * 30),    # velocity, psi, rho, mu, kappa, p in; velocity out
        "projection": (2 * nd + 5, (2 * nd + 3) * 2 * 30),         # psi, p, rho, velocity in; kappa, div, velocity out
    }.get(kind, (3, 20))                                           # a solve: right-hand side, density in; pressure out
    return {"bytes": 8.0 * fields * n, "flops": float(flops) * n}


# ---- the same in 64 bits ----------------------------------------------------------------------
def _ccd_matrices(n, periodic):
    """Dense (D1, D2) of the sixth-order combined compact scheme on n + 1 nodes of a unit axis,
    f' + (7/16)(f'_- + f'_+) - (h/16)(f''_+ - f''_-) = (15/16)(f_+ - f_-)/h and
    f'' - (1/8)(f''_- + f''_+) + (9/8)(f'_+ - f'_-)/h = 3 (f_+ - 2 f + f_-)/h^2,
    with one-sided wall closures or periodic wrap-around."""
    h, m = 1.0 / n, n + 1
    u = n if periodic else m
    A = torch.zeros(2 * u, 2 * u, dtype=torch.float64)
    B = torch.zeros(2 * u, u, dtype=torch.float64)
    for i in range(u):
        A[2 * i, 2 * i] = A[2 * i + 1, 2 * i + 1] = 1.0
        if not periodic and i in (0, n):
            s, j = (1, 1) if i == 0 else (-1, n - 1)
            A[2 * i, 2 * j], A[2 * i, 2 * j + 1] = 1.5, -1.5 * h * s
            for k, c in enumerate((-23.0 / 6.0, 21.0 / 4.0, -1.5, 1.0 / 12.0)):
                B[2 * i, i + s * k] += s * c / h
            for k, c in enumerate((45.0, -154.0, 214.0, -156.0, 61.0, -10.0)):
                B[2 * i + 1, i + s * k] += c / (12.0 * h * h)
            continue
        lo, hi = ((i - 1) % u, (i + 1) % u) if periodic else (i - 1, i + 1)
        for j, s in ((lo, 1.0), (hi, -1.0)):
            A[2 * i, 2 * j] += 7.0 / 16.0
            A[2 * i, 2 * j + 1] += s * h / 16.0
            A[2 * i + 1, 2 * j] += -s * 9.0 / (8.0 * h)
            A[2 * i + 1, 2 * j + 1] += -1.0 / 8.0
        B[2 * i, hi] += 15.0 / (16.0 * h)
        B[2 * i, lo] -= 15.0 / (16.0 * h)
        B[2 * i + 1, lo] += 3.0 / (h * h)
        B[2 * i + 1, hi] += 3.0 / (h * h)
        B[2 * i + 1, i] -= 6.0 / (h * h)
    X = torch.linalg.solve(A.to(_dev()), B.to(_dev()))
    D1, D2 = X[0::2], X[1::2]
    if periodic:   # the image node stores node 0's value and is not read
        D1, D2 = (torch.cat([torch.cat([D, D[:1]]), torch.zeros(m, 1, dtype=D.dtype, device=D.device)], 1)
                  for D in (D1, D2))
    return D1.contiguous(), D2.contiguous()


class _Exact:
    """CCD derivatives of FP64 fields by dense matrices."""

    def __init__(self, N, bc="wall"):
        self.N, self.nd, self.periodic = N, len(N), bc == "periodic"
        made = {n: _ccd_matrices(n, self.periodic) for n in set(N)}
        self.D = [made[n] for n in N]
        self.h = [1.0 / n for n in N]

    def along(self, M, f, ax):
        g = f.movedim(ax, 0)
        return (M @ g.reshape(g.shape[0], -1)).reshape(M.shape[0], *g.shape[1:]).movedim(0, ax).contiguous()

    def d1(self, f, ax):
        return self.along(self.D[ax][0], f, ax)

    def d2(self, f, ax):
        return self.along(self.D[ax][1], f, ax)

    def sync(self, f):
        return _sync_images(f) if self.periodic else f

    def slab(self, f, ax, a, b):
        return f.narrow(ax, a, b - a)


def _exact_flux(x, u, phi, ax):
    """-d(u phi)/dx by face values (p_L + p_R)/2 - (h^2/16)(q_L + q_R), q the CCD second derivative."""
    N, h = x.N[ax], x.h[ax]
    p = u * phi
    q = x.d2(p, ax)
    lo, hi = (x.slab(t, ax, 0, N) for t in (p, q)), (x.slab(t, ax, 1, N + 1) for t in (p, q))
    (pl, ql), (pr, qr) = lo, hi
    face = 0.5 * (pl + pr) - (h * h / 16.0) * (ql + qr)
    out = torch.zeros_like(p)
    if x.periodic:
        d = (face - torch.roll(face, 1, ax)) / h
        x.slab(out, ax, 0, N).copy_(d)
        out.select(ax, N).copy_(d.select(ax, 0))
    else:
        x.slab(out, ax, 1, N).copy_((x.slab(face, ax, 1, N) - x.slab(face, ax, 0, N - 1)) / h)
    return -out


def _exact_mass_fix(q, dV, target):
    w = 4.0 * q * (1.0 - q)
    W = (w * dV).sum()
    return torch.clamp(q + (target - (q * dV).sum()) / W * w, 0.0, 1.0)


def _exact_volumes(x):
    """Control volumes: h per axis on walls; no volume on a periodic image node."""
    vol = torch.ones([1] * x.nd, dtype=torch.float64, device=_dev())
    for ax in range(x.nd):
        w = torch.full((x.N[ax] + 1,), x.h[ax], dtype=torch.float64, device=_dev())
        if x.periodic:
            w[-1] = 0.0
        vol = vol * _along(w, ax, x.nd)
    return vol.expand([n + 1 for n in x.N])


def _exact_levelset(case, s):
    x = _Exact(_cells(case), case["bc"])
    nd, dt, vel, q0 = x.nd, s["dt"], s["vel"], s["psi"]
    dV = _exact_volumes(x)

    def stage(q):
        return q + dt * sum(_exact_flux(x, vel[k], q, k) for k in range(nd))

    def keep(q):
        return x.sync(torch.clamp(q, 0.0, 1.0))

    q = keep(stage(q0))
    q = keep(0.75 * q0 + 0.25 * stage(q))
    q = keep(q0 / 3.0 + 2.0 / 3.0 * stage(q))
    moved = x.sync(_exact_mass_fix(q, dV, (q0 * dV).sum()))
    # reinitialization: 4 pseudo-steps of compression (forward Euler) and Crank-Nicolson diffusion
    eps, dx = 1.5 / max(x.N), min(x.h)
    dtau = min(0.5 * dx * dx / (2.0 * nd * eps), 0.5 * dx)
    q = moved.clone()
    cn = []
    for ax in range(nd):
        n, mu = x.N[ax] + 1, eps * dtau / (2.0 * x.h[ax] ** 2)
        A, B = (torch.zeros(n, n, dtype=torch.float64, device=_dev()) for _ in range(2))
        for M, d, c in ((A, 1.0 + 6.0 * mu, -0.125 - 3.0 * mu), (B, 1.0 - 6.0 * mu, -0.125 + 3.0 * mu)):
            M.diagonal().fill_(d)
            M.diagonal(1).fill_(c)
            M.diagonal(-1).fill_(c)
            M[0, 1] = M[n - 1, n - 2] = 2.0 * c
        cn.append(torch.linalg.solve(A, B))
    for _ in range(4):
        g = [x.d1(q, ax) for ax in range(nd)]
        norm = torch.clamp(torch.sqrt(torch.clamp(sum(t * t for t in g), min=1e-12)), min=1e-6)
        div = torch.zeros_like(q)
        for ax in range(nd):
            d = x.d1(q * (1.0 - q) * (g[ax] / norm), ax)
            n = x.N[ax] + 1
            first, last = (n - 2, 1) if x.periodic else (0, n - 1)
            pad = torch.cat([x.slab(d, ax, first, first + 1), d, x.slab(d, ax, last, last + 1)], ax)
            div += d + 0.05 * (x.slab(pad, ax, 2, n + 2) - 2.0 * d + x.slab(pad, ax, 0, n))
        q = keep(q - dtau * div)
        for ax in range(nd):
            q = x.sync(x.along(cn[ax], q, ax))
        q = keep(q)
    return {"moved": moved, "sharp": x.sync(_exact_mass_fix(q, dV, (moved * dV).sum()))}


def _exact_low(x, f, ax):
    """Second-order first derivative, one-sided at the ends."""
    n, h, out = x.N[ax] + 1, x.h[ax], torch.empty_like(f)
    x.slab(out, ax, 1, n - 1).copy_((x.slab(f, ax, 2, n) - x.slab(f, ax, 0, n - 2)) / (2.0 * h))
    out.select(ax, 0).copy_((f.select(ax, 1) - f.select(ax, 0)) / h)
    out.select(ax, n - 1).copy_((f.select(ax, n - 1) - f.select(ax, n - 2)) / h)
    return out


def _exact_grad_p(x, p):
    out = []
    for ax in range(x.nd):
        g = x.d1(p, ax)
        g.select(ax, 0).zero_()
        g.select(ax, x.N[ax]).zero_()
        out.append(g)
    return out


def _exact_predictor(case, s):
    x = _Exact(_cells(case))
    nd, u, rho, mu, dt = x.nd, s["vel"], s["rho"], s["mu"], s["dt"]

    def viscous(v):
        G = [[x.d1(v[a], b) for b in range(nd)] for a in range(nd)]
        return [sum(_exact_low(x, mu * (G[a][b] + G[b][a]), b) for b in range(nd)) / (REYNOLDS * rho)
                for a in range(nd)]

    gp = _exact_grad_p(x, s["p"])
    e = []
    for c in range(nd):
        conv = torch.zeros_like(rho)
        for k in range(nd):
            if case["convection"] == "uccd6":
                d8 = x.d2(x.d2(x.d2(x.d2(u[c], k), k), k), k)
                conv -= 0.5 * (u[k] * x.d1(u[c], k) + x.d1(u[k] * u[c], k))
                conv -= 1e-3 * x.h[k] ** 7 * u[k].abs().max() * d8
            else:
                conv -= u[k] * x.d1(u[c], k)
        t = rho * conv + s["kappa"] * x.d1(s["psi"], c) / WEBER - gp[c]
        e.append(t - rho / FROUDE ** 2 if c == nd - 1 else t)
    vn = viscous(u)
    vs = viscous([u[c] + dt * (e[c] / rho + vn[c]) for c in range(nd)])
    return [u[c] + dt * (e[c] / rho + 0.5 * vn[c] + 0.5 * vs[c]) for c in range(nd)]


def _exact_curvature(x, psi):
    nd, sw = x.nd, (2.0 * psi - 1.0) ** 2

    def smooth(f):
        out = f
        for ax in range(nd):
            n, prev = x.N[ax] + 1, out
            out = prev.clone()
            c = x.slab(prev, ax, 1, n - 1)
            x.slab(out, ax, 1, n - 1).add_(0.05 * x.slab(sw, ax, 1, n - 1)
                                           * (x.slab(prev, ax, 2, n) - 2.0 * c + x.slab(prev, ax, 0, n - 2)))
        for ax in range(nd):
            for k in (0, x.N[ax]):
                out.select(ax, k).copy_(f.select(ax, k))
        return out

    g = [smooth(x.d1(psi, ax)) for ax in range(nd)]
    gg = [smooth(x.d2(psi, ax)) for ax in range(nd)]
    sq = sum(t * t for t in g) + 1e-30
    if nd == 2:
        xy = smooth(x.d1(g[0], 1))
        k = -(g[1] * g[1] * gg[0] - 2.0 * g[0] * g[1] * xy + g[0] * g[0] * gg[1]) / sq ** 1.5
    else:
        con = sum(g[a] * g[a] * gg[a] for a in range(3))
        con = con + sum(2.0 * g[i] * g[j] * x.d1(g[i], j) for i in range(3) for j in range(i + 1, 3))
        k = -(sum(gg) - con / sq) / torch.sqrt(sq)
    return torch.where((psi <= 0.01) | (psi >= 0.99), torch.zeros_like(k), k)


def _exact_projection(case, s):
    x = _Exact(_cells(case))
    p, rho, dt = s["p"], s["rho"], s["dt"]
    div = torch.zeros_like(p)
    for ax in range(x.nd):
        n, h, u = x.N[ax] + 1, x.h[ax], s["vel"][ax]
        dp = x.d1(p, ax)
        dp.select(ax, 0).copy_((p.select(ax, 1) - p.select(ax, 0)) / h)
        dp.select(ax, n - 1).copy_((p.select(ax, n - 1) - p.select(ax, n - 2)) / h)
        (ul, pl, rl, dl), (ur, pr, rr, dr) = ([x.slab(t, ax, a, a + n - 1) for t in (u, p, rho, dp)] for a in (0, 1))
        face = 0.5 * (ul + ur) - dt * 2.0 / (rl + rr) * ((pr - pl) / h - 0.5 * (dl + dr))
        edge = torch.zeros_like(x.slab(face, ax, 0, 1))
        flux = torch.cat([edge, face, edge], ax)
        div += (x.slab(flux, ax, 1, n + 1) - x.slab(flux, ax, 0, n)) / h
    gp = _exact_grad_p(x, p)
    return {"kappa": _exact_curvature(x, s["psi"]), "div": div,
            "vel": [s["vel"][a] - dt / rho * gp[a] for a in range(x.nd)]}


def _exact_solve(N, rhs, rho):
    """p with p = 0 at the middle node and div(grad p / rho) = rhs at every other node (finite
    volumes, zero normal gradient on walls): Jacobi-preconditioned CG to round-off."""
    nd = len(N)
    width = []
    for n in N:
        w = torch.full((n + 1,), 1.0 / n, dtype=torch.float64, device=rhs.device)
        w[0] = w[-1] = 0.5 / n
        width.append(w)
    vol = torch.ones([1] * nd, dtype=torch.float64, device=rhs.device)
    for ax in range(nd):
        vol = vol * _along(width[ax], ax, nd)
    free = torch.ones_like(rhs)
    free[tuple(n // 2 for n in N)] = 0.0
    coup = []
    for ax, n in enumerate(N):
        c = 2.0 * n / (rho.narrow(ax, 0, n) + rho.narrow(ax, 1, n))
        for b in range(nd):
            if b != ax:
                c = c * _along(width[b], b, nd)
        coup.append(c)

    def spread(parts):
        out = torch.zeros_like(rhs)
        for ax, n in enumerate(N):
            out.narrow(ax, 0, n).sub_(parts[ax][0])
            out.narrow(ax, 1, n).add_(parts[ax][1])
        return out

    diag = spread([(-c, c) for c in coup])

    def mul(p):
        f = [coup[ax] * (p.narrow(ax, 1, n) - p.narrow(ax, 0, n)) for ax, n in enumerate(N)]
        return spread([(t, t) for t in f]) * free

    b = -(rhs * vol) * free
    x = torch.zeros_like(b)
    stop = 1e-13 * torch.linalg.vector_norm(b)
    for _ in range(3):   # restarted on the true residual
        r = b - mul(x)
        z = r / diag * free
        p, rz = z.clone(), (r * z).sum()
        for it in range(20000):
            q = mul(p)
            a = rz / (p * q).sum()
            x += a * p
            r -= a * q
            if it % 50 == 49 and bool(torch.linalg.vector_norm(r) < stop):
                break
            z = r / diag * free
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
        if bool(torch.linalg.vector_norm(b - mul(x)) < 4.0 * stop):
            break
    return x


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "ccd":
        x, f = _Exact(_cells(case), case["bc"]), s["f"].double()
        return [(x.d1(f, ax), x.d2(f, ax)) for ax in range(x.nd)]
    if kind == "levelset":
        return _exact_levelset(case, s)
    if kind == "predictor":
        return _exact_predictor(case, s)
    if kind == "projection":
        return _exact_projection(case, s)
    if kind == "batch":
        return [_exact_solve(n, y["rhs"], y["rho"]) for n, y in zip(_batch_grids(case), s["systems"])]
    return _exact_solve(_cells(case), s["rhs"], s["rho"])
