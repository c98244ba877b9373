"""Workloads of the Stokes solver, the stochastic fluxes and the timesteps, as
a simulation program calls them, for timing one version of the library against
another.

Five kinds, over the sizes the library is used at (2D 48^2 to 512^2, 3D 24^3 to
256^3, uneven extents among them), in both precisions:

  gmres   one preconditioned solve of the staggered Stokes system
  step    one inertial timestep of a mixture with freshly drawn noise
  batch   overdamped steps of many 2D realizations of uneven size
  stoch   the stochastic momentum flux divergence
  mass    the diffusive and stochastic mass flux divergence of a mixture

`listed` gives the named cases, `draw` one more of the same ranges, `prepare`
what a program holds before the call, `run` one pass, `work` the bytes and
operations the pass needs at least, and `exact` the results in 64 bits by
plain torch where there is a closed form.
"""
from __future__ import annotations

import math

import torch

import lowmachfhd_b200 as L

F64 = torch.float64
DEV = "cuda"
MOLMASS = [1.0, 2.0, 3.0, 4.0, 5.0]
KT = 1e-4


def listed():
    g = dict(kind="gmres", nz=1, visc=1, walls=False, dense=False)
    return [
        # the smallest solve: one overdamped Stokes solve on a 64^2 grid, plain
        # FP64; latency and launches are all of it
        dict(g, name="gmres_2d_64_fp64", dim=2, nx=64, ny=64, precision="fp64", theta=0.0, dx=1.0, tol=1e-9),
        # the largest served 2D request's solve
        dict(g, name="gmres_2d_512_mixed", dim=2, nx=512, ny=512, precision="mixed", theta=0.0, dx=1.0, tol=1e-8),
        # a channel between no-slip walls
        dict(g, name="gmres_2d_channel_mixed", dim=2, nx=256, ny=128, precision="mixed", theta=10.0, dx=1.0,
             tol=1e-8, walls=True),
        # a small served 3D request's solve; 40 = 8 * 5 coarsens to 5^3 only
        dict(g, name="gmres_3d_40_mixed", dim=3, nx=40, ny=40, nz=40, precision="mixed", theta=0.2, dx=10.0,
             tol=1e-8),
        # variable viscosity with the symmetric stress (visc_type -2) and
        # variable density, uneven box, plain FP64
        dict(g, name="gmres_3d_varvisc_fp64", dim=3, nx=96, ny=64, nz=80, visc=-2, precision="fp64", theta=0.2,
             dx=10.0, tol=1e-8, dense=True),
        # the solve of the 128^3 fluctuating Navier-Stokes run in plain FP64
        dict(g, name="gmres_3d_128_fp64", dim=3, nx=128, ny=128, nz=128, precision="fp64", theta=20.0, dx=1.0,
             tol=1e-9),
        # the largest served 3D request's solve, variable density
        dict(g, name="gmres_3d_192_mixed", dim=3, nx=192, ny=192, nz=192, precision="mixed", theta=0.2, dx=10.0,
             tol=1e-8, dense=True),
        # the headline workload: one step of the 4-species mixture at 256^3
        dict(name="step_3d_256_4sp_mixed", kind="step", nx=256, ny=256, nz=256, ns=4, precision="mixed"),
        # a served step of ordinary size
        dict(name="step_3d_64_2sp_mixed", kind="step", nx=64, ny=64, nz=64, ns=2, precision="mixed"),
        # a batch of realizations of uneven size
        dict(name="batch_2d_128_boxes", kind="batch", boxes=128, lo=32, hi=256, precision="mixed", steps=1),
        # the symmetric stochastic stress of a 192^3 run
        dict(name="stoch_3d_192_mixed", kind="stoch", dim=3, nx=192, ny=192, nz=192, precision="mixed", sym=True,
             rngs=1),
        # the mass fluxes of the 4-species mixture
        dict(name="mass_3d_128_4sp_mixed", kind="mass", dim=3, nx=128, ny=128, nz=128, ns=4, precision="mixed"),
    ]


def _log(rng, lo, hi, mult=1):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / mult)) * mult))


def draw(rng):
    prec = rng.choice(["mixed", "mixed", "fp64"])
    kind = rng.choice(["gmres", "gmres", "gmres", "step", "batch", "stoch", "mass"])
    if kind == "gmres":
        # sides are multiples of 8, as served requests round them; the odd
        # multiples coarsen to odd bottoms
        dim = rng.choice([2, 3])
        lo, hi = (48, 512) if dim == 2 else (24, 128)
        nx, ny = _log(rng, lo, hi, 8), _log(rng, lo, hi, 8)
        nz = _log(rng, lo, hi, 8) if dim == 3 else 1
        walls = rng.random() < 0.2
        return dict(kind="gmres", dim=dim, nx=nx, ny=ny, nz=nz, visc=1 if walls else rng.choice([1, 1, 1, -1, -2, 2]),
                    precision=prec, theta=rng.choice([0.0, 1.0, 20.0]) if dim == 2 else rng.choice([0.2, 20.0]),
                    dx=1.0 if dim == 2 else 10.0, tol=rng.choice([1e-8, 1e-9]), walls=walls,
                    dense=rng.random() < 0.5)
    if kind == "step":
        n = _log(rng, 24, 96, 8)
        return dict(kind="step", nx=n, ny=_log(rng, 24, 96, 8), nz=n, ns=rng.choice([2, 3, 4]), precision=prec)
    if kind == "batch":
        return dict(kind="batch", boxes=_log(rng, 4, 96), lo=32, hi=rng.choice([64, 128, 200]), precision=prec,
                    steps=1)
    dim = rng.choice([2, 3, 3])
    lo, hi = (65, 1024) if dim == 2 else (17, 160)
    nx, ny = _log(rng, lo, hi), _log(rng, lo, hi)
    nz = _log(rng, lo, hi) if dim == 3 else 1
    if kind == "stoch":
        return dict(kind="stoch", dim=dim, nx=nx, ny=ny, nz=nz, precision=prec, sym=rng.random() < 0.6,
                    rngs=rng.choice([1, 2]))
    return dict(kind="mass", dim=dim, nx=nx, ny=ny, nz=nz, ns=rng.choice([2, 3, 4]), precision=prec)


# ----------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _cells(case):
    return [case["nx"], case["ny"], case["nz"]][: case.get("dim", 3)]


def _mixture(ns, seed):
    """masses 1..ns, Maxwell-Stefan coefficients U[0.5, 2] * 1e-2"""
    g = torch.Generator().manual_seed(1000 + int(seed))
    D = ((0.5 + 1.5 * torch.rand(ns * (ns - 1) // 2, generator=g, dtype=F64)) * 1e-2).tolist()
    return MOLMASS[:ns], D


def _gmres_inputs(case, seed):
    """right-hand side and coefficients: a white random force as the
    stochastic stress gives it, a divergence constraint of zero mean"""
    g, dim, n = _gen(seed), case["dim"], _cells(case)
    nc = math.prod(n)
    nE = 1 if dim == 2 else 3
    rnd = lambda: torch.randn(nc, generator=g, dtype=F64, device=DEV)
    b_u = [rnd() for _ in range(dim)]
    b_u = [b - b.mean() for b in b_u] if case["theta"] == 0.0 else b_u
    b_p = 1e-2 * rnd()
    b_p -= b_p.mean()
    if case["walls"]:
        # the normal force on a wall face is zero
        b_u[1].view(n[::-1])[..., 0, :] = 0.0
    one = torch.ones(nc, dtype=F64, device=DEV)
    # face densities of a mixture with a few per cent of fluctuation
    alpha = [1.0 + 0.03 * rnd().clamp(-5, 5) for _ in range(dim)] if case["dense"] else [one] * dim
    if case["visc"] < 0:
        beta = 1.0 + 0.5 * torch.rand(nc, generator=g, dtype=F64, device=DEV)
        bed = [1.0 + 0.5 * torch.rand(nc, generator=g, dtype=F64, device=DEV) for _ in range(nE)]
    else:
        beta, bed = one, [one] * nE
    return b_u, b_p, alpha, beta, bed, torch.zeros_like(one)


def _stoch_inputs(case, seed):
    g, dim = _gen(seed), case["dim"]
    nc = math.prod(_cells(case))
    nE = 1 if dim == 2 else 3
    rnd = lambda: torch.randn(nc, generator=g, dtype=F64, device=DEV)
    W_cc, W_ed = [], []
    for _ in range(case["rngs"]):
        # the symmetric form: cell entries of variance 2, the two components
        # of an edge equal
        W_cc += [rnd() * (math.sqrt(2.0) if case["sym"] else 1.0) for _ in range(dim)]
        for _ in range(nE):
            e = rnd()
            W_ed += [e, e if case["sym"] else rnd()]
    var = lambda: 1.0 + 0.2 * torch.rand(nc, generator=g, dtype=F64, device=DEV)
    eta, T = var(), var()
    return eta, [var() for _ in range(nE)], T, [var() for _ in range(nE)], W_cc, W_ed


def _mass_inputs(case, seed):
    g, ns, dim = _gen(seed), case["ns"], case["dim"]
    nc = math.prod(_cells(case))
    w = 1.0 / ns + 0.02 * torch.randn(ns, nc, generator=g, dtype=F64, device=DEV).clamp(-5, 5)
    w /= w.sum(dim=0, keepdim=True)
    W = [torch.randn(nc, generator=g, dtype=F64, device=DEV) for _ in range(dim * ns)]
    return [w[i].contiguous() for i in range(ns)], W


class _State:
    """what the program keeps: a context, its stream and the fields"""


def prepare(case, seed):
    s = _State()
    s.kind = kind = case["kind"]
    if kind == "batch":
        u = torch.rand(case["boxes"], generator=torch.Generator().manual_seed(case["boxes"]), dtype=F64)
        eta = torch.rand(case["boxes"], generator=torch.Generator().manual_seed(int(seed)), dtype=F64)
        lo, hi = math.log(case["lo"]), math.log(case["hi"])
        # the batch's square sides log-uniform, multiples of 8 without the odd multiples
        # above 13, whose 8-smooth bottoms would set the pace of all boxes
        sides = [int(round(math.exp(lo + (hi - lo) * float(x)) / 8)) * 8 for x in u]
        sides = [n if (n // 8) % 2 == 0 or n // 8 <= 13 else n - 8 for n in sides]
        s.B = L.Batch([(n, n) for n in sides], 1.0, params=L.default_params(gmres_rel_tol=1e-8),
                      precision=case["precision"])
        s.u = [torch.zeros(s.B.total, dtype=F64, device=DEV) for _ in range(2)]
        s.pi = torch.zeros(s.B.total, dtype=F64, device=DEV)
        s.eta = [0.5 + 4.5 * float(x) for x in eta]
        s.kT = [1.0] * case["boxes"]
        s.steps, s.seed, s.step0 = case["steps"], int(seed), 0
        torch.cuda.synchronize()
        return s
    n = _cells(case)
    s.dim = dim = len(n)
    nc = math.prod(n)
    nE = 1 if dim == 2 else 3
    s.stream = torch.cuda.Stream()
    new = lambda k: [torch.zeros(nc, dtype=F64, device=DEV) for _ in range(k)]
    if kind == "gmres":
        s.theta = case["theta"]
        s.b_u, s.b_p, s.alpha, s.beta, s.bed, s.gamma = _gmres_inputs(case, seed)
        s.x_u, (s.x_p,) = new(dim), new(1)
        kw = dict(bc_lo=[-1, 100, -1][:dim], bc_hi=[-1, 100, -1][:dim]) if case["walls"] else {}
        s.ctx = L.StokesSolver(dim, n, case["dx"], case["visc"], params=L.default_params(gmres_rel_tol=case["tol"]),
                               precision=case["precision"], **kw)
    else:
        s.dx = 10.0 if dim == 3 else 1.0
        s.dt = 5.0 if dim == 3 else 0.1
        s.ctx = L.StokesSolver(dim, n, s.dx, 1, params=L.default_params(gmres_rel_tol=1e-8),
                               precision=case["precision"])
        s.sp = L.StochParams(k_B=KT, variance_coef_mom=1.0, dV=1000.0, stoch_stress_form=1, filtering_width=0)
    s.ctx.set_stream(s.stream.cuda_stream)
    if kind == "stoch":
        s.sp.stoch_stress_form = 1 if case["sym"] else 0
        s.eta, s.eta_ed, s.T, s.T_ed, s.W_cc, s.W_ed = _stoch_inputs(case, seed)
        s.weights = [1.0] if case["rngs"] == 1 else [math.sqrt(0.5)] * 2
        s.out = new(dim)
    elif kind == "mass":
        s.rho, s.W = _mass_inputs(case, seed)
        mm, D = _mixture(case["ns"], seed)
        s.mp = L.mixture_params(mm, D)
        s.out = new(case["ns"])
    elif kind == "step":
        ns = case["ns"]
        g = _gen(seed)
        mm, D = _mixture(ns, seed)
        s.mp = L.mixture_params(mm, D)
        w = 1.0 / ns + 1e-3 * torch.randn(ns, nc, generator=g, dtype=F64, device=DEV)
        w /= w.sum(dim=0, keepdim=True)
        s.state0 = [1e-3 * torch.randn(nc, generator=g, dtype=F64, device=DEV) for _ in range(dim)]
        s.state0 += [w[i].contiguous() for i in range(ns)] + new(1)
        s.state = [t.clone() for t in s.state0]
        s.F0, s.F = new(ns), new(ns)
        one = torch.ones(nc, dtype=F64, device=DEV)
        s.eta, s.eta_ed, s.T, s.T_ed, (s.kappa,) = one, [one] * nE, one, [one] * nE, new(1)
        s.noise = L.StepNoise(dim, n, ns, int(seed), DEV, stream=s.stream.cuda_stream)
        s.ns = ns
        torch.cuda.synchronize()
        # F^0, the mass fluxes of the initial state
        s.noise.draw_mass(0)
        s.ctx.compute_mass_fluxdiv(s.mp, s.sp, s.state0[dim:dim + ns], s.dt, [1.0], s.noise.mass(0), s.F0)
    torch.cuda.synchronize()
    return s


# ----------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------
def run(s):
    if s.kind == "batch":
        # the next steps of every realization, in place
        s.B.overdamped(s.u, s.pi, s.eta, s.kT, 0.1, s.steps, seed=s.seed, step0=s.step0)
        s.step0 += s.steps
        return s.u + [s.pi]
    if s.kind == "gmres":
        with torch.cuda.stream(s.stream):
            for t in s.x_u + [s.x_p]:
                t.zero_()
        s.ctx.gmres(s.b_u, s.b_p, s.x_u, s.x_p, s.alpha, s.beta, s.bed, s.gamma, s.theta)
        return s.x_u + [s.x_p]
    if s.kind == "stoch":
        s.ctx.stochastic_m_fluxdiv(s.sp, s.out, False, s.eta, s.eta_ed, s.T, s.T_ed, s.dt, s.weights, s.W_cc, s.W_ed)
        return s.out
    if s.kind == "mass":
        s.ctx.compute_mass_fluxdiv(s.mp, s.sp, s.rho, s.dt, [1.0], s.W, s.out)
        return s.out
    # the first step of a realization from the stored initial state (its M_0
    # stays in the noise ring; the step's own fields are drawn)
    with torch.cuda.stream(s.stream):
        for t, t0 in zip(s.state + s.F, s.state0 + s.F0):
            t.copy_(t0)
    s.noise.draw(1)
    W_cc, W_ed, W_mass = s.noise.inertial_args(1)
    u, rho, pi = s.state[: s.dim], s.state[s.dim: s.dim + s.ns], s.state[-1]
    s.ctx.advance_timestep_inertial_multispecies(s.sp, s.mp, s.dt, u, rho, pi, s.F, s.eta, s.eta_ed, s.kappa, s.T,
                                                 s.T_ed, W_cc, W_ed, W_mass)
    return s.state + s.F


# ----------------------------------------------------------------------
# least work
# ----------------------------------------------------------------------
def _solve_flops(nc, dim):
    """four iterations (the fewest that reach 1e-8 here), each one operator
    application, one V-cycle of each multigrid (four smooths and a residual
    per level) and the orthogonalisation"""
    vcycle = 5 * (dim * (4 * dim + 4) + 6 * dim) * (8.0 / 7.0 if dim == 3 else 4.0 / 3.0)
    return 4.0 * nc * (vcycle + dim * (4 * dim + 6) + 10 * (dim + 1))


def work(case):
    kind = case["kind"]
    if kind == "batch":
        nc = case["boxes"] * (case["hi"] ** 2 - case["lo"] ** 2) / (2 * math.log(case["hi"] / case["lo"]))
        return {"bytes": 8.0 * nc * 6 * case["steps"], "flops": 2 * case["steps"] * _solve_flops(nc, 2)}
    n = _cells(case)
    dim, nc = len(n), float(math.prod(n))
    nE = 1 if dim == 2 else 3
    if kind == "gmres":
        words = 2 * (dim + 1) + dim + (1 + nE if case["visc"] < 0 else 0)
        return {"bytes": 8.0 * nc * words, "flops": _solve_flops(nc, dim)}
    if kind == "stoch":
        ed = nE if case["sym"] else 2 * nE
        words = case["rngs"] * (dim + ed) + 2 * (1 + nE) + dim
        return {"bytes": 8.0 * nc * words, "flops": nc * (4.0 * (dim + ed) * case["rngs"] + 6 * dim)}
    ns = case["ns"]
    chi = 10 * 2 * ns ** 3 + 20 * ns ** 2
    mass = {"bytes": 8.0 * nc * (ns + dim * ns + ns), "flops": nc * (chi + dim * (chi + ns ** 3 + 8 * ns ** 2))}
    if kind == "mass":
        return mass
    words = 2 * (dim + 2 * ns + 1) + (dim + nE + dim * ns)
    return {"bytes": 8.0 * nc * words, "flops": 2 * mass["flops"] + 2 * _solve_flops(nc, dim)}


# ----------------------------------------------------------------------
# results in 64 bits
# ----------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "gmres":
        return _exact_gmres(case, seed)
    if case["kind"] == "stoch":
        return _exact_stoch(case, seed)
    if case["kind"] == "mass":
        return _exact_mass(case, seed)
    return None


def _exact_gmres(case, seed):
    """the constant-coefficient periodic system, mode by mode:
    lam u_d + g_d p = b_d, sum_d conj(g_d) u_d = b_p"""
    if case["walls"] or case["dense"] or case["visc"] != 1:
        return None
    b_u, b_p, *_ = _gmres_inputs(case, seed)
    n, dx, theta = _cells(case)[::-1], case["dx"], case["theta"]
    dim = len(n)
    k = torch.meshgrid(*[2 * math.pi * torch.fft.fftfreq(m, dtype=F64, device=DEV) for m in n], indexing="ij")[::-1]
    g = [(1.0 - torch.exp(-1j * q)) / dx for q in k]
    gg = sum(x.abs() ** 2 for x in g)
    lam = theta + gg
    B = [torch.fft.fftn(b.view(n)) for b in b_u]
    P = torch.fft.fftn(b_p.view(n))
    gg0, lam0 = gg.clone(), lam.clone()
    gg0.view(-1)[0] = 1.0
    if theta == 0.0:
        lam0.view(-1)[0] = 1.0
    p = (sum(x.conj() * b for x, b in zip(g, B)) - lam * P) / gg0
    p.view(-1)[0] = 0.0
    out = []
    for d in range(dim):
        u = (B[d] - g[d] * p) / lam0
        if theta == 0.0:
            u.view(-1)[0] = 0.0
        out.append(torch.fft.ifftn(u).real.reshape(-1))
    return out + [torch.fft.ifftn(p).real.reshape(-1)]


def _exact_stoch(case, seed):
    eta, eta_ed, T, T_ed, W_cc, W_ed = _stoch_inputs(case, seed)
    n = _cells(case)[::-1]
    dim = len(n)
    nE = 1 if dim == 2 else 3
    dx, dt = (10.0, 5.0) if dim == 3 else (1.0, 0.1)
    wt = [1.0] if case["rngs"] == 1 else [math.sqrt(0.5)] * 2
    var = math.sqrt(2.0 * KT / (1000.0 * dt))
    lo = lambda a, d: a - torch.roll(a, 1, dims=dim - 1 - d)
    hi = lambda a, d: torch.roll(a, -1, dims=dim - 1 - d) - a
    cc = [var * sum(w * W_cc[r * dim + c] for r, w in enumerate(wt)) * (eta * T).sqrt() for c in range(dim)]
    ed = [[var * sum(w * W_ed[2 * (r * nE + e) + q] for r, w in enumerate(wt)) * (eta_ed[e] * T_ed[e]).sqrt()
           for q in range(2)] for e in range(nE)]
    cc = [a.view(n) for a in cc]
    ed = [[a.view(n) for a in e] for e in ed]
    out = []
    for c in range(dim):
        f = lo(cc[c], c)
        for d in range(dim):
            if d != c:
                a, b = min(c, d), max(c, d)
                e = 0 if dim == 2 or (a, b) == (0, 1) else 1 if (a, b) == (0, 2) else 2
                f = f + hi(ed[e][0 if c < d else 1], d)
        out.append((f / dx).reshape(-1))
    return out


def _exact_mass(case, seed):
    rho, W = _mass_inputs(case, seed)
    mm, Dl = _mixture(case["ns"], seed)
    ns, n = case["ns"], _cells(case)[::-1]
    dim = len(n)
    dx, dt, dV = (10.0, 5.0, 1000.0) if dim == 3 else (1.0, 0.1, 1000.0)
    D, k = [[0.0] * ns for _ in range(ns)], 0
    for r in range(ns):
        for c in range(r):
            D[r][c] = D[c][r] = Dl[k]
            k += 1

    def conc(r):
        rt = sum(r)
        w = [a / rt for a in r]
        mt = 1.0 / sum(a / m for a, m in zip(w, mm))
        return rt, w, mt, [mt * a / m for a, m in zip(w, mm)]

    def chi(r):
        rt, w, mt, x = conc(r)
        if ns == 2:
            t = mm[0] * w[1] + mm[1] * w[0]
            t = D[0][1] * t * t / (mm[0] * mm[1])
            return [[t * w[1] / w[0], -t], [-t, t * w[0] / w[1]]]
        mw = sum(a * m for a, m in zip(x, mm))
        Y = [m * a / mw for a, m in zip(x, mm)]
        t2 = [sum(x[j] / D[i][j] for j in range(ns) if j != i) for i in range(ns)]
        Di = [(1.0 - Y[i]) / t2[i] for i in range(ns)]
        Minv = [Di[i] / x[i] for i in range(ns)]
        J = [[Minv[i] * (x[i] / Di[i] - x[i] * t2[i] if i == j else x[i] * x[j] / D[i][j]) for j in range(ns)]
             for i in range(ns)]
        cs = [sum(Y[q] * J[q][j] for q in range(ns)) for j in range(ns)]
        PJ = [[J[i][j] - cs[j] for j in range(ns)] for i in range(ns)]
        sY = sum(Y[q] * Y[q] * Minv[q] for q in range(ns))
        m2 = [[(Minv[i] if i == j else 0.0) - Y[i] * Minv[i] - Y[j] * Minv[j] + sY for j in range(ns)]
              for i in range(ns)]
        X = m2
        for _ in range(10):
            X = [[m2[i][j] + sum(PJ[i][q] * X[q][j] for q in range(ns)) for j in range(ns)] for i in range(ns)]
        return X

    rho = [a.view(n) for a in rho]
    rwc = [[rho[i] * c for c in row] for i, row in enumerate(chi(rho))]
    x = conc(rho)[3]
    out = [torch.zeros_like(rho[0]) for _ in range(ns)]
    var = math.sqrt(2.0 * KT / (dV * dt))
    for d in range(dim):
        ax = dim - 1 - d
        m = lambda a: torch.roll(a, 1, dims=ax)
        gx = [(a - m(a)) / dx for a in x]
        f = [sum(0.5 * (m(rwc[r][c]) + rwc[r][c]) * gx[c] for c in range(ns)) for r in range(ns - 1)]
        ra = []
        for s_, a in enumerate(rho):
            v1, v2 = m(a) / mm[s_], a / mm[s_]
            o = mm[s_] * (v1 + v2) / 2 * (dV * v1).clamp(max=1.0) * (dV * v2).clamp(max=1.0)
            ra.append(torch.where((v1 <= 0) | (v2 <= 0), torch.zeros_like(o), o))
        rt, w, mt, _ = conc(ra)
        ch = chi(ra)
        A = [[mt * rt * w[r] * ch[r][c] * w[c] / KT for c in range(ns)] for r in range(ns)]
        # Cholesky rows but the last, whose flux is minus the sum of the others
        C = [[None] * ns for _ in range(ns)]
        for i in range(ns - 1):
            for j in range(i + 1):
                t = A[i][j] - sum(C[i][q] * C[j][q] for q in range(j))
                C[i][j] = t.clamp(min=0.0).sqrt() if i == j else t / C[j][j]
        for r in range(ns - 1):
            f[r] = f[r] + var * sum(C[r][c] * W[d * ns + c].view(n) for c in range(r + 1))
        f.append(-sum(f))
        for s_ in range(ns):
            out[s_] += (torch.roll(f[s_], -1, dims=ax) - f[s_]) / dx
    return [a.reshape(-1) for a in out]
