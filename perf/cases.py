"""The work that users of this package have it do, as cases with sizes.

``listed()`` gives the fixed cases, ``draw()`` more of the same kinds and
ranges, ``prepare()`` what a program holds before the call, ``run()`` one pass
through the public entry points, ``exact()`` the same outputs from plain torch
in 64 bits.  The package computes in FP64 throughout, so ``exact()`` is a
second implementation of the scheme rather than a more precise one: the
finite-difference right-hand side, the stages, the ghost fill of uniform
meshes, the ADM maps, the constraints, psi4, and the reverse mode of a step by
torch's autograd.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gr-athena_b200"))
import z4c_b200 as Z  # noqa: E402

NG = 4
# 1+log / Gamma-driver gauge, constraint damping and Kreiss-Oliger strength of
# the puncture runs; the gauge wave's harmonic-like gauge
PUNCTURE = dict(diss=0.02, chi_div_floor=1e-5, damp_kappa1=0.02, damp_kappa2=0.0, shift_eta=2.0,
                r_max_con=1e300)
WAVE = dict(lapse_harmonic=1.0, lapse_harmonicf=0.0, lapse_oplog=0.0, lapse_advect=0.0,
            shift_Gamma=0.0, shift_eta=0.0, shift_advect=0.0, diss=0.02, damp_kappa1=0.02,
            r_max_con=1e300)


def listed():
    return [
        # one right-hand side of one MeshBlock: an operator called from a host
        # program's own time loop, where latency counts
        dict(name="rhs_block", kind="rhs", bx=1, by=1, bz=1, nx=16, ny=16, nz=16, bc="periodic",
             contract=False),
        # the same on a few blocks of odd sizes, contracted arithmetic
        dict(name="rhs_ragged", kind="rhs", bx=3, by=2, bz=2, nx=22, ny=13, nz=18, bc="outflow",
             contract=True),
        # the gauge-wave convergence run: one 48^3 block, a few steps at a time
        dict(name="evolve_wave", kind="evolve", bx=1, by=1, bz=1, nx=48, ny=48, nz=48,
             bc="periodic", contract=False, integ="rk4", steps=4, con=False),
        # the uniform puncture mesh on the default path, constraints for the
        # history file after the step
        dict(name="evolve_puncture", kind="evolve", bx=8, by=8, bz=8, nx=16, ny=16, nz=16,
             bc="outflow", contract=False, integ="rk4", steps=1, con=True),
        # the same mesh in production: contracted arithmetic, several steps a call
        dict(name="evolve_contracted", kind="evolve", bx=8, by=8, bz=8, nx=16, ny=16, nz=16,
             bc="outflow", contract=True, integ="rk4", steps=4, con=False),
        # radiative boundaries with the classical integrator, larger blocks
        dict(name="evolve_sommerfeld", kind="evolve", bx=4, by=3, bz=2, nx=24, ny=24, nz=24,
             bc="sommerfeld", contract=False, integ="bt_rk4", steps=1, con=True),
        # a binary on nested refinement boxes with its puncture trackers
        dict(name="refined_binary", kind="refined", root=4, levels=4, contract=True, steps=1),
        # constraint monitoring of a state: ADM variables, constraints, norms
        dict(name="diagnostics", kind="diagnostics", bx=8, by=8, bz=4, nx=16, ny=16, nz=16,
             bc="outflow"),
        # initial data: ADM variables to the evolved ones, ghosts filled
        dict(name="initial_data", kind="initial", bx=4, by=4, bz=4, nx=32, ny=32, nz=32,
             bc="outflow"),
        # wave extraction after a step: psi4, its ghosts, two spheres
        dict(name="psi4", kind="psi4", bx=4, by=4, bz=4, nx=16, ny=16, nz=16, bc="outflow",
             nlev=10, lmax=4),
        # one reverse step of a gradient run
        dict(name="adjoint", kind="adjoint", bx=1, by=1, bz=1, nx=40, ny=40, nz=40,
             bc="periodic"),
        # a parameter sweep whose states live in host memory
        dict(name="jobs", kind="jobs", bx=4, by=4, bz=4, nx=16, ny=16, nz=16, bc="outflow",
             contract=True, jobs=3, steps=1),
    ]


def draw(rng):
    """One more case: kinds in turn by chance, sizes over the logarithm of
    their range, most of them odd."""
    kind = rng.choice(["rhs", "rhs", "evolve", "evolve", "evolve", "refined", "diagnostics",
                       "initial", "psi4", "adjoint", "jobs"])
    if kind == "refined":
        return dict(kind=kind, root=rng.choice([2, 3, 4]), levels=rng.randint(1, 4),
                    contract=rng.random() < 0.5, steps=1)
    cap = {"rhs": 2.1e6, "evolve": 2.1e6, "diagnostics": 1.05e6, "initial": 2.1e6,
           "psi4": 2.6e5, "adjoint": 6.4e4, "jobs": 2.6e5}[kind]
    goal = math.exp(rng.uniform(math.log(6e3), math.log(cap)))
    while True:
        b = [rng.choice([1, 1, 2, 3, 4, 5, 8]) for _ in range(3)]
        n = [rng.choice([16, rng.randint(8, 24), rng.randint(8, 48)]) for _ in range(3)]
        if rng.random() < 0.4:
            n = [16, 16, 16]
        zones = math.prod(b) * math.prod(n)
        if 0.6 * goal <= zones <= min(1.4 * goal, cap):
            break
    case = dict(kind=kind, bx=b[0], by=b[1], bz=b[2], nx=n[0], ny=n[1], nz=n[2],
                bc=rng.choice(["periodic", "outflow"]))
    if kind in ("rhs", "evolve"):
        case["contract"] = rng.random() < 0.5
    if kind == "evolve":
        if rng.random() < 0.3:
            case.update(bc="sommerfeld", contract=False)
        case.update(integ="bt_rk4" if rng.random() < 0.2 else "rk4", con=rng.random() < 0.5,
                    steps=rng.randint(1, 3) if zones < 7e5 else 1)
    elif kind == "psi4":
        case.update(nlev=rng.randint(3, 12), lmax=rng.randint(2, 4))
    elif kind == "adjoint":
        case.update(bc="periodic")
    elif kind == "jobs":
        case.update(contract=True, jobs=rng.randint(1, 3), steps=rng.randint(1, 2))
    return case


# ---- meshes and states -------------------------------------------------------

def _wave_like(case):
    return case.get("bc") == "periodic"


def _params(case):
    p = dict(WAVE if _wave_like(case) and case["kind"] == "evolve" else PUNCTURE)
    if case["kind"] == "adjoint":
        p["eps_floor"] = -1.0  # the differentiable constraint projection
    return p


def _mesh(case):
    if case["kind"] == "refined":
        half = 16.0
        boxes = []
        for lev in range(1, case["levels"] + 1):
            r = half / 2 ** lev
            boxes.append({**{f"x{a}min": -r * (1.2 if a == 1 else 0.7) for a in (1, 2, 3)},
                          **{f"x{a}max": r * (1.2 if a == 1 else 0.7) for a in (1, 2, 3)},
                          "level": lev})
        return Z.Mesh((case["root"],) * 3, (16,) * 3, (-half,) * 3, (half,) * 3, "outflow",
                      refinement=boxes)
    nb, nx = (case["bx"], case["by"], case["bz"]), (case["nx"], case["ny"], case["nz"])
    h = _spacing(case)
    lo = tuple(-0.5 * b * n * h * f for b, n, f in zip(nb, nx, (1.0, 1.1, 0.9)))
    return Z.Mesh(nb, nx, lo, tuple(-v for v in lo), case["bc"])


def _spacing(case):
    n = max(case["bx"] * case["nx"], case["by"] * case["ny"], case["bz"] * case["nz"])
    return (1.0 if _wave_like(case) else 12.0) / n


def _coords(case, mesh):
    """Vertex coordinates, ghosts included, as broadcastable (x, y, z) with a
    leading block axis; a vertex shared by blocks gets the same value in each."""
    out = []
    for a in range(3):
        nn, nx = mesh.nn[a], mesh.nx[a]
        i = torch.arange(nn, dtype=torch.float64, device="cuda") - NG
        if mesh.locs is None:
            nb = mesh.nb
            b = torch.arange(mesh.nblocks, device="cuda")
            lo = (b % nb[0], (b // nb[0]) % nb[1], b // (nb[0] * nb[1]))[a]
            scale = torch.ones(mesh.nblocks, dtype=torch.float64, device="cuda")
        else:
            locs = torch.as_tensor(np.asarray(mesh.locs), device="cuda")
            lo = locs[:, 1 + a]
            scale = 2.0 ** (locs[:, 0] - mesh.root_level).double()
        span = mesh.xmax[a] - mesh.xmin[a]
        g = lo.double()[:, None] * nx + i[None, :]
        x = mesh.xmin[a] + g * (span / (mesh.nb[a] * nx)) / scale[:, None]
        shape = [mesh.nblocks, 1, 1, 1]
        shape[3 - a] = nn
        out.append(x.reshape(shape))
    return out


def _state(case, mesh, seed, member=0):
    """A smooth Z4c state [block][22][k][j][i], the algebraic constraints
    satisfied: on periodic meshes a superposition of waves of per cent
    amplitude around flat space, otherwise two punctures with the collapsed
    lapse and per cent perturbations that fall off outwards."""
    rng = random.Random(1000003 * seed + member)
    X, Y, W = _coords(case, mesh)
    ones = torch.ones_like(X * Y * W)
    u = torch.empty((mesh.nblocks, 22) + tuple(reversed(mesh.nn)), dtype=torch.float64,
                    device="cuda")
    base = [0.0] * 22
    for v in (Z.CHI, Z.GXX, Z.GYY, Z.GZZ, Z.ALPHA):
        base[v] = 1.0
    wave = case["kind"] != "refined" and _wave_like(case)
    if wave:
        span = [mesh.xmax[a] - mesh.xmin[a] for a in range(3)]
        amp, psi, fall = 0.01, None, None
    else:
        amp = 0.02
        psi = ones.clone()
        for s in (1.0, -1.0):
            m = rng.uniform(0.4, 0.6)
            c = (s * rng.uniform(1.0, 1.6), rng.uniform(-0.3, 0.3), rng.uniform(-0.3, 0.3))
            psi += 0.5 * m / ((X - c[0]) ** 2 + (Y - c[1]) ** 2 + (W - c[2]) ** 2
                              + 1e-6).sqrt()
        fall = torch.exp(-(X * X + Y * Y + W * W) / 18.0)
    for v in range(22):
        f = torch.zeros_like(ones)
        for _ in range(2):
            if wave:
                k = [2 * math.pi * rng.randint(-2, 2) / span[a] for a in range(3)]
            else:
                k = [rng.uniform(-1.0, 1.0) for _ in range(3)]
            f += rng.uniform(0.3, 1.0) * torch.sin(k[0] * X + k[1] * Y + k[2] * W
                                                   + rng.uniform(0, 2 * math.pi))
        f *= amp
        if fall is not None:
            f *= fall
        if psi is not None and v == Z.CHI:
            u[:, v] = psi ** -4 * (1.0 + f)
        elif psi is not None and v == Z.ALPHA:
            u[:, v] = psi ** -2 * (1.0 + f)
        else:
            u[:, v] = base[v] + f
    return _alg_constr(u, -1.0)


class _Register:
    """Register `reg` of a context through the CUDA array interface; a tensor
    made from it holds this object and so keeps the context alive."""

    def __init__(self, ctx, reg):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": ctx.shape(reg), "typestr": "<f8", "version": 3,
                                         "data": (ctx.device_ptr(reg), False)}


def _view(ctx, reg):
    """Register `reg` of the context as a torch tensor on the same memory."""
    return torch.as_tensor(_Register(ctx, reg), device="cuda")


def _adm_data(case, mesh, seed):
    """ADM variables of a smooth perturbed binary [block][17][k][j][i]."""
    return _z4c_to_adm(_state(case, mesh, seed))


def prepare(case, seed):
    mesh = _mesh(case)
    ctx = Z.Z4c(mesh, Z.default_params(**_params(case)), case.get("integ", "rk4"))
    s = {"case": case, "ctx": ctx}
    if case.get("contract"):
        ctx.set_contract(True)
    kind = case["kind"]
    torch.cuda.synchronize()
    if kind == "initial":
        _view(ctx, Z.REG_ADM).copy_(_adm_data(case, mesh, seed))
        torch.cuda.synchronize()
        return s
    if kind == "jobs":
        shape = ctx.shape(Z.REG_U)
        s["in"] = []
        for j in range(case["jobs"]):
            _view(ctx, Z.REG_U).copy_(_state(case, mesh, seed, j))
            torch.cuda.synchronize()
            ctx.Z4cToADM()
            ctx.init_finalize()
            ctx.sync()
            s["in"].append(torch.empty(shape, dtype=torch.float64, pin_memory=True))
            s["in"][j].copy_(_view(ctx, Z.REG_U))
        s["out"] = [torch.empty(shape, dtype=torch.float64, pin_memory=True)
                    for _ in range(case["jobs"])]
        s["dt"] = 0.25 * min(ctx.dx())
        torch.cuda.synchronize()
        return s
    _view(ctx, Z.REG_U).copy_(_state(case, mesh, seed))
    torch.cuda.synchronize()
    ctx.Z4cToADM()
    ctx.init_finalize()
    if kind == "refined":
        for x in (1.3, -1.3):
            ctx.add_tracker((x + 0.01, 0.013, 0.017))
        s["dt"] = mesh.new_dt(0.25)
    else:
        s["dt"] = 0.25 * min(ctx.dx())
    if kind == "psi4":
        r = 0.3 * (mesh.xmax[0] - mesh.xmin[0]) * min(
            1.0, *[(mesh.xmax[a] - mesh.xmin[a]) / (mesh.xmax[0] - mesh.xmin[0])
                   for a in (1, 2)])
        s["spheres"] = [Z.WaveExtract(ctx, radius=f * r, nlev=case["nlev"], lmax=case["lmax"])
                        for f in (0.8, 1.4)]
    if kind == "adjoint":
        ctx.adj_setup()
        ctx.sync()
        _view(ctx, Z.REG_ADJ).copy_(_cotangent(ctx.shape(Z.REG_ADJ), seed))
        torch.cuda.synchronize()
    ctx.sync()
    return s


def _cotangent(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 77)
    return torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "rhs":
        ctx.Z4cRHS()
        return {"rhs": _view(ctx, Z.REG_RHS)}
    if kind in ("evolve", "refined"):
        con = bool(case.get("con"))
        ctx.evolve(s["dt"], case["steps"], con)
        out = {"u": _view(ctx, Z.REG_U), "adm": _view(ctx, Z.REG_ADM)}
        if con:
            out["con"] = _view(ctx, Z.REG_CON)
        if kind == "refined":
            out["trackers"] = np.concatenate([np.concatenate(ctx.tracker(t)) for t in (0, 1)])
        return out
    if kind == "diagnostics":
        ctx.constraints()
        return {"norms": ctx.hst_norms(), "adm": _view(ctx, Z.REG_ADM),
                "con": _view(ctx, Z.REG_CON)}
    if kind == "initial":
        ctx.ADMToZ4c()
        ctx.init_finalize()
        return {"u": _view(ctx, Z.REG_U), "adm": _view(ctx, Z.REG_ADM)}
    if kind == "psi4":
        psi = ctx.psi4_multipoles(s["spheres"])
        return {"weyl": _view(ctx, Z.REG_WEYL), "inner": psi[0], "outer": psi[1]}
    if kind == "adjoint":
        ctx.adj_step(s["dt"])
        return {"ubar": _view(ctx, Z.REG_ADJ)}
    norms = ctx.evolve_jobs([a.numpy() for a in s["in"]], [a.numpy() for a in s["out"]], s["dt"],
                            case["steps"])
    return {"norms": norms, **{f"u{j}": a for j, a in enumerate(s["out"])}}


# ---- what a pass cannot do without -------------------------------------------

def _points(case):
    """(interior vertices, all vertices) of the mesh."""
    if case["kind"] == "refined":
        n = _mesh(case).nblocks
        return n * 17 ** 3, n * 25 ** 3
    b = case["bx"] * case["by"] * case["bz"]
    n = (case["nx"], case["ny"], case["nz"])
    return b * math.prod(v + 1 for v in n), b * math.prod(v + 9 for v in n)


def work(case):
    """Bytes: every input register read once and every output written once;
    a stage reads u and u1 and writes both (the Butcher stages u, u_n and the
    slope).  Operations: 7,697 per interior vertex and right-hand side and 154
    per stage update, counted with a counting number type; the other kinds
    scaled from their own counts."""
    inner, every = _points(case)
    kind = case["kind"]
    stage = 4 * (704 * inner), 4 * (7851 * inner)
    con = (8 * (11 * inner + 7 * every), 6000 * inner) if case.get("con") else (0, 0)
    if kind == "rhs":
        return {"bytes": 8 * 22 * (inner + every), "flops": 7697 * inner}
    if kind in ("evolve", "refined"):
        n = case["steps"]
        return {"bytes": n * (stage[0] + 8 * 17 * every) + con[0], "flops": n * stage[1] + con[1]}
    if kind == "diagnostics":
        return {"bytes": 8 * (22 + 17 + 7) * every, "flops": 6000 * inner}
    if kind == "initial":
        return {"bytes": 8 * (17 + 22) * every, "flops": 250 * every}
    if kind == "psi4":
        return {"bytes": 8 * (22 + 17 + 2) * every, "flops": 7409 * inner}
    if kind == "adjoint":
        return {"bytes": 4 * 3 * 8 * 22 * every, "flops": 4 * 3 * 7851 * inner}
    n = case["jobs"]
    return {"bytes": n * (case["steps"] * stage[0] + 2 * 8 * 22 * every),
            "flops": n * case["steps"] * stage[1]}


def tolerance(case):
    """FP64 throughout.  Each bound is about four times (more where the meshes
    drawn are finer or step longer) what the contracted path differs from the
    exact one, another order of the same sums, or either from the plain-torch
    values.  On meshes with outflow or Sommerfeld faces three cascades of
    five-point extrapolations multiply rounding in the corner ghosts by up to
    1e9; these carry the largest single differences there."""
    kind = case["kind"]
    if kind in ("evolve", "jobs", "initial") and case["bc"] == "periodic":
        return {"rel": 1e-10, "max": 1e-8}
    return {"rhs": {"rel": 1e-11, "max": 3e-10}, "evolve": {"rel": 4e-9, "max": 1e-5},
            "refined": {"rel": 5e-10, "max": 1e-6}, "diagnostics": {"rel": 1e-11, "max": 3e-10},
            "initial": {"rel": 1e-9, "max": 3e-6}, "psi4": {"rel": 3e-7, "max": 2e-4},
            "adjoint": {"rel": 1e-13, "max": 1e-12},
            "jobs": {"rel": 2e-9, "max": 4e-6}}[kind]


# ---- the same scheme in plain torch ------------------------------------------

PAIRS = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))
SYM = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
R3 = range(3)
D1 = (-1 / 60, 9 / 60, -45 / 60, 0.0, 45 / 60, -9 / 60, 1 / 60)
D2 = (2 / 180, -27 / 180, 270 / 180, -490 / 180, 270 / 180, -27 / 180, 2 / 180)
KO = (1, -8, 28, -56, 70, -56, 28, -8, 1)
LEFT = (1, -8, 30, -80, 35, 24, -2)          # offsets -4..2
RIGHT = (2, -24, -35, 80, -30, 8, -1)        # offsets -2..4


def _sym(f):
    """3x3 lists from the six stored components."""
    return [[f[SYM[a][b]] for b in R3] for a in R3]


def _crop(f, d):
    """f without d vertices at each end of (x, y, z)."""
    return f[..., d[2]:f.shape[-3] - d[2], d[1]:f.shape[-2] - d[1], d[0]:f.shape[-1] - d[0]]


def _conv(f, a, c, first, half):
    """sum_q c[q] f(i + first + q) along axis a, for the vertices that are at
    least `half` from both ends of that axis."""
    dim = -1 - a
    n = f.shape[dim] - 2 * half
    return sum(w * f.narrow(dim, half + first + q, n) for q, w in enumerate(c) if w)


def _d(f, a, h):
    d = [4, 4, 4]
    d[a] = 1
    return _conv(_crop(f, d), a, D1, -3, 3) / h[a]


def _dd(f, a, b, h):
    d = [4, 4, 4]
    if a == b:
        d[a] = 1
        return _conv(_crop(f, d), a, D2, -3, 3) / h[a] ** 2
    d[a] = d[b] = 1
    return _conv(_conv(_crop(f, d), b, D1, -3, 3), a, D1, -3, 3) / (h[a] * h[b])


def _axis(f, a):
    d = [4, 4, 4]
    d[a] = 0
    return _crop(f, d)


def _advect(f, beta, h):
    out = 0
    for a in R3:
        g = _axis(f, a)
        out = out + beta[a] / (60 * h[a]) * torch.where(
            beta[a] < 0, _conv(g, a, LEFT, -4, 4), _conv(g, a, RIGHT, -2, 4))
    return out


def _det(g):
    return (g[0][0] * (g[1][1] * g[2][2] - g[1][2] ** 2)
            - g[0][1] * (g[0][1] * g[2][2] - g[1][2] * g[0][2])
            + g[0][2] * (g[0][1] * g[1][2] - g[1][1] * g[0][2]))


def _inv(g):
    d = _det(g)
    i = [(g[1][1] * g[2][2] - g[1][2] ** 2) / d, (g[0][2] * g[1][2] - g[0][1] * g[2][2]) / d,
         (g[0][1] * g[1][2] - g[0][2] * g[1][1]) / d, (g[0][0] * g[2][2] - g[0][2] ** 2) / d,
         (g[0][1] * g[0][2] - g[0][0] * g[1][2]) / d, (g[0][0] * g[1][1] - g[0][1] ** 2) / d]
    return _sym(i)


def _christoffel(dg, gu):
    """(first kind [c][a][b], second kind) from dg[c][a][b] = d_c g_ab."""
    lo = [[[0.5 * (dg[a][b][c] + dg[b][a][c] - dg[c][a][b]) for b in R3] for a in R3] for c in R3]
    up = [[[sum(gu[c][d] * lo[d][a][b] for d in R3) for b in R3] for a in R3] for c in R3]
    return lo, up


def _rhs(u, p, h, som=None):
    """Right-hand side on the interior, Kreiss-Oliger included."""
    I = [_crop(u[:, v], (4, 4, 4)) for v in range(22)]
    F = [u[:, v] for v in range(22)]
    g, A = _sym(I[1:7]), _sym(I[8:14])
    chi, Kh, Th, al = I[0].clamp(min=p.chi_div_floor), I[7], I[17], I[18]
    Gam, beta = I[14:17], I[19:22]
    gu = _inv(g)
    dg = [_sym([_d(F[1 + q], c, h) for q in range(6)]) for c in R3]
    G, Gu = _christoffel(dg, gu)
    Gc = [sum(gu[b][c] * Gu[a][b][c] for b in R3 for c in R3) for a in R3]
    dGam = [[_d(F[14 + c], b, h) for c in R3] for b in R3]
    dchi = [_d(F[0], a, h) for a in R3]
    dal = [_d(F[18], a, h) for a in R3]
    db = [[_d(F[19 + a], b, h) for a in R3] for b in R3]
    dphi = [-dchi[a] / (4 * chi) for a in R3]
    DDphi = _sym([-_dd(F[0], a, b, h) / (4 * chi) + 4 * dphi[a] * dphi[b]
                  - sum(Gu[c][a][b] * dphi[c] for c in R3) for a, b in PAIRS])
    S = sum(gu[a][b] * (DDphi[a][b] + 2 * dphi[a] * dphi[b]) for a in R3 for b in R3)
    R = []
    for q, (a, b) in enumerate(PAIRS):
        r = sum(0.5 * (g[c][a] * dGam[b][c] + g[c][b] * dGam[a][c]
                       + Gc[c] * (G[a][b][c] + G[b][a][c])) for c in R3)
        r = r - 0.5 * sum(gu[c][d] * _dd(F[1 + q], min(c, d), max(c, d), h)
                          for c in R3 for d in R3)
        r = r + sum(gu[c][d] * (Gu[e][c][a] * G[b][e][d] + Gu[e][c][b] * G[a][e][d]
                                + Gu[e][a][d] * G[e][c][b])
                    for c in R3 for d in R3 for e in R3)
        R.append(r + 4 * dphi[a] * dphi[b] - 2 * DDphi[a][b] - 2 * g[a][b] * S)
    R = _sym(R)
    ww = sum(gu[c][d] * dphi[c] * dal[d] for c in R3 for d in R3)
    DDal = _sym([_dd(F[18], a, b, h) - 2 * (dphi[a] * dal[b] + dphi[b] * dal[a])
                 + 2 * g[a][b] * ww - sum(Gu[c][a][b] * dal[c] for c in R3) for a, b in PAIRS])
    lap = sum(chi * gu[a][b] * DDal[a][b] for a in R3 for b in R3)
    Aud = [[sum(gu[a][c] * A[c][b] for c in R3) for b in R3] for a in R3]
    AA = [[sum(A[a][c] * Aud[c][b] for c in R3) for b in R3] for a in R3]
    trAA = sum(gu[a][b] * AA[a][b] for a in R3 for b in R3)
    Au = [[sum(gu[b][c] * Aud[a][c] for c in R3) for b in R3] for a in R3]
    K = Kh + 2 * Th
    dK, dT = [_d(F[7], a, h) for a in R3], [_d(F[17], a, h) for a in R3]
    DA = [sum(-1.5 * Au[a][b] * dchi[b] / chi - gu[a][b] * (2 * dK[b] + dT[b]) / 3 for b in R3)
          + sum(Gu[a][b][c] * Au[b][c] for b in R3 for c in R3) for a in R3]
    Rs = sum(chi * gu[a][b] * R[a][b] for a in R3 for b in R3)
    Ht = Rs + 2 / 3 * K * K - trAA
    div = db[0][0] + db[1][1] + db[2][2]
    ddb = [[[_dd(F[19 + c], min(a, b), max(a, b), h) for b in R3] for a in R3] for c in R3]
    ddiv = [sum(ddb[b][a][b] for b in R3) / 3 for a in R3]
    L = [_advect(F[v], beta, h) for v in range(22)]
    out = [None] * 22
    out[0] = L[0] - 2 / 3 * chi * div + 2 / 3 * chi * al * K
    out[7] = -lap + al * (trAA + K * K / 3) + L[7] + p.damp_kappa1 * (1 - p.damp_kappa2) * al * Th
    out[17] = L[17] + al * (0.5 * Ht - (2 + p.damp_kappa2) * p.damp_kappa1 * Th)
    for a in R3:
        lg = L[14 + a] + 2 / 3 * Gc[a] * div + sum(
            gu[a][b] * ddiv[b] - Gc[b] * db[b][a] for b in R3) + sum(
            gu[b][c] * ddb[a][b][c] for b in R3 for c in R3)
        out[14 + a] = 2 * al * DA[a] + lg - 2 * al * p.damp_kappa1 * (Gam[a] - Gc[a]) - sum(
            2 * Au[a][b] * dal[b] for b in R3)
        out[19 + a] = p.shift_Gamma * Gam[a] + p.shift_advect * L[19 + a] - p.shift_eta * beta[a]
    for q, (a, b) in enumerate(PAIRS):
        lg = L[1 + q] - 2 / 3 * g[a][b] * div + sum(
            db[a][c] * g[b][c] + db[b][c] * g[a][c] for c in R3)
        la = L[8 + q] - 2 / 3 * A[a][b] * div + sum(
            db[b][c] * A[a][c] + db[a][c] * A[b][c] for c in R3)
        out[1 + q] = -2 * al * A[a][b] + lg
        out[8 + q] = (chi * (-DDal[a][b] + al * R[a][b]) - g[a][b] * (-lap + al * Rs) / 3
                      + al * (K * A[a][b] - 2 * AA[a][b]) + la)
    out[18] = p.lapse_advect * L[18] - (p.lapse_oplog * p.lapse_harmonicf
                                        + p.lapse_harmonic * al) * al * (Kh + 2 * p.lapse_K * Th)
    for v in range(22):
        out[v] = out[v] + sum(_conv(_axis(F[v], a), a, KO, -4, 4) * (-p.diss / (256 * h[a]))
                              for a in R3)
    out = torch.stack(out, 1)
    return out if som is None else som(u, out)


def _sommerfeld(case, mesh, h):
    """Sommerfeld condition on the outer vertex planes."""
    X = [_crop(x.expand(mesh.nblocks, *reversed(mesh.nn)), (4, 4, 4)) for x in _coords(case, mesh)]
    r = (X[0] ** 2 + X[1] ** 2 + X[2] ** 2).sqrt()
    on = torch.zeros_like(r, dtype=torch.bool)
    for a in R3:
        e = 1e-9 * h[a]
        on |= (X[a] < mesh.xmin[a] + e) | (X[a] > mesh.xmax[a] - e)

    def apply(u, out):
        out = out.clone()
        for v in (7, 17) + tuple(range(8, 17)):
            c = math.sqrt(2.0) if v == 7 else 1.0
            f = u[:, v]
            w = _crop(f, (4, 4, 4)) / r
            for a in R3:
                d = [4, 4, 4]
                d[a] = 3
                w = w + X[a] / r * _conv(_crop(f, d), a, (-0.5, 0.0, 0.5), -1, 1) / h[a]
            out[:, v] = torch.where(on, -c * w, out[:, v])
        return out
    return apply


def _alg_constr(u, eps):
    """det g~ = 1 (left as it is within eps above 1, as the package does) and
    tr A~ = 0, at every vertex."""
    v = list(u.unbind(1))
    g = _sym(v[1:7])
    d = _det(g)
    d = torch.where(d > 0, d, torch.ones_like(d))
    s = torch.where(d - 1.0 < eps, torch.full_like(d, 1.0 - eps / 3.0), d ** (-1 / 3))
    v[1:7] = [x * s for x in v[1:7]]
    g, A = _sym(v[1:7]), _sym(v[8:14])
    d = _det(g)
    adj = _inv(g)
    tr = sum(d * adj[a][b] * A[a][b] for a in R3 for b in R3)
    v[8:14] = [v[8 + q] - tr * v[1 + q] / 3 for q in range(6)]
    # vertices no fill writes hold zeros, where the inverse does not exist
    out = torch.stack(v, 1)
    return torch.where(torch.isfinite(out), out, u)


def _fill(w, mesh):
    """Ghost fill of a uniform mesh from the blocks' interiors: owners'
    average on shared vertices, neighbours' values in the ghosts, then the
    extrapolation of non-periodic faces."""
    nb, nx, nn = mesh.nb, mesh.nx, mesh.nn
    periodic = mesh.bc[0] == Z.BC_PERIODIC
    size = [nb[a] * nx[a] + (0 if periodic else 1) for a in R3]
    b = torch.arange(mesh.nblocks, device="cuda")
    loc = (b % nb[0], (b // nb[0]) % nb[1], b // (nb[0] * nb[1]))

    def index(a, lo, hi):
        i = loc[a][:, None] * nx[a] + torch.arange(lo, hi, device="cuda")[None, :]
        ok = torch.ones_like(i, dtype=torch.bool) if periodic else (i >= 0) & (i < size[a])
        return (i % size[a] if periodic else i.clamp(0, size[a] - 1)), ok

    own = [index(a, 0, nx[a] + 1)[0] for a in R3]
    flat = ((own[2][:, :, None, None] * size[1] + own[1][:, None, :, None]) * size[0]
            + own[0][:, None, None, :]).reshape(-1)
    n = size[0] * size[1] * size[2]
    inner = _crop(w, (4, 4, 4)).transpose(0, 1).reshape(w.shape[1], -1)
    total = torch.zeros((w.shape[1], n), dtype=w.dtype, device=w.device).index_add(1, flat, inner)
    count = torch.zeros(n, dtype=w.dtype, device=w.device).index_add(
        0, flat, torch.ones(flat.numel(), dtype=w.dtype, device=w.device))
    mean = total / count
    at, ok = zip(*[index(a, -NG, nx[a] + 1 + NG) for a in R3])
    flat = ((at[2][:, :, None, None] * size[1] + at[1][:, None, :, None]) * size[0]
            + at[0][:, None, None, :])
    inside = (ok[2][:, :, None, None] & ok[1][:, None, :, None] & ok[0][:, None, None, :])
    out = (mean[:, flat.reshape(-1)].reshape((w.shape[1],) + tuple(flat.shape)).transpose(0, 1)
           * inside[:, None])
    if periodic:
        return out
    out = out.contiguous()
    where = [v.tolist() for v in loc]
    for a in R3:
        for side in (0, 1):
            for blk in range(mesh.nblocks):
                l = [where[c][blk] for c in R3]
                if l[a] != (nb[a] - 1 if side else 0):
                    continue
                r = [slice(0, 2 * NG + nx[c]) for c in R3]
                for c in (1, 2):
                    if c != a and not (a == 2 and c == 1):
                        r[c] = slice(NG if l[c] == 0 else 0,
                                     NG + nx[c] if l[c] == nb[c] - 1 else 2 * NG + nx[c])
                v = out[blk].movedim(3 - a, 0)
                rest = [r[c] for c in (2, 1, 0) if c != a]
                for q in range(NG):
                    i, d = (NG + nx[a] + q, -1) if side else (NG - 1 - q, 1)
                    v[(i, slice(None), *rest)] = sum(
                        c * v[(i + d * (m + 1), slice(None), *rest)]
                        for m, c in enumerate((5.0, -10.0, 10.0, -5.0, 1.0)))
    return out


def _pad(f):
    return torch.nn.functional.pad(f, (4,) * 6)


def _step(u, p, h, mesh, dt, integ="rk4", som=None, stage_wrap=lambda f, *x: f(*x)):
    """One RK4 step of the whole register; fills read interiors only, so the
    stage values carry zeros in the ghosts."""
    if integ == "rk4":
        gam = ((0.0, 1.0), (0.121098479554482, 0.721781678111411),
               (-3.843833699660025, 2.121209265338722), (0.546370891121863, 0.198653035682705))
        delta = (1.0, 0.217683334308543, 1.065841341361089, 0.0)
        bdt = (1.193743905974738, 0.099279895495783, 1.131678018054042, 0.310665766509336)
        v = torch.zeros_like(_crop(u, (4, 4, 4)))
        for s in range(4):
            def stage(u, v, s=s):
                i = _crop(u, (4, 4, 4))
                v = v + delta[s] * i
                w = gam[s][0] * i + gam[s][1] * v + bdt[s] * dt * _rhs(u, p, h, som)
                return _alg_constr(_fill(_pad(w), mesh), p.eps_floor), v
            u, v = stage_wrap(stage, u, v)
        return u
    un, ks = _crop(u, (4, 4, 4)), []
    for c in (0.5, 0.5, 1.0, None):
        ks.append(_rhs(u, p, h, som))
        w = un + dt * (c * ks[-1] if c else (ks[0] + 2 * ks[1] + 2 * ks[2] + ks[3]) / 6)
        u = _alg_constr(_fill(_pad(w), mesh), p.eps_floor)
    return u


def _z4c_to_adm(u):
    psi4 = torch.where(u[:, 0] != 0, 1.0 / u[:, 0], torch.full_like(u[:, 0], math.inf))
    K = (u[:, 7] + 2 * u[:, 17]) / 3
    out = [u[:, 18], u[:, 19], u[:, 20], u[:, 21]] + [psi4 * u[:, 1 + q] for q in range(6)]
    out += [psi4 * u[:, 8 + q] + K * psi4 * u[:, 1 + q] for q in range(6)]
    return torch.stack(out + [psi4], 1)


def _adm_to_z4c(adm, h):
    G, K = _sym([adm[:, 4 + q] for q in range(6)]), _sym([adm[:, 10 + q] for q in range(6)])
    s = _det(G) ** (-1 / 3)
    g = [s * G[a][b] for a, b in PAIRS]
    gu = _inv(_sym(g))
    tr = sum(gu[a][b] * s * K[a][b] for a in R3 for b in R3)
    A = [s * K[a][b] - tr * g[q] / 3 for q, (a, b) in enumerate(PAIRS)]
    z = torch.zeros_like(s)
    Gam = [_pad(-sum(_d(gu[b][a], b, h) for b in R3)[:, None])[:, 0] for a in R3]
    return torch.stack([s] + g + [tr] + A + Gam + [z] + [adm[:, v] for v in range(4)], 1)


def _curvature(u, adm, p, h):
    """Physical metric, its inverse, Christoffels, Ricci tensor, K_ab, D_a K_bc
    on the interior, the metric's derivatives by the chain rule from those of
    the conformal metric and chi."""
    I = [_crop(u[:, v], (4, 4, 4)) for v in range(22)]
    chi = I[0].clamp(min=p.chi_div_floor)
    gt = _sym(I[1:7])
    dchi = [_d(u[:, 0], a, h) for a in R3]
    dgt = [_sym([_d(u[:, 1 + q], c, h) for q in range(6)]) for c in R3]
    J = [_crop(adm[:, v], (4, 4, 4)) for v in range(17)]
    g, K = _sym(J[4:10]), _sym(J[10:16])
    gu = _inv(g)
    dg = [[[(dgt[c][a][b] - gt[a][b] * dchi[c] / chi) / chi for b in R3] for a in R3] for c in R3]
    ddg = {}
    for a, b in PAIRS:
        ddc = _dd(u[:, 0], a, b, h)
        for q, (c, d) in enumerate(PAIRS):
            v = (_dd(u[:, 1 + q], a, b, h)
                 - (dchi[a] * dgt[b][c][d] + dchi[b] * dgt[a][c][d] + ddc * gt[c][d]) / chi
                 + 2 * dchi[a] * dchi[b] * gt[c][d] / chi ** 2) / chi
            for x, y in ((a, b), (b, a)):
                ddg[x, y, c, d] = ddg[x, y, d, c] = v
    G, Gu = _christoffel(dg, gu)
    R = _sym([sum(gu[c][d] * sum(Gu[e][a][c] * G[e][b][d] - Gu[e][a][b] * G[e][c][d] for e in R3)
                  for c in R3 for d in R3)
              + 0.5 * sum(gu[c][d] * (-ddg[c, d, a, b] - ddg[a, b, c, d] + ddg[a, c, b, d]
                                      + ddg[b, c, a, d]) for c in R3 for d in R3)
              for a, b in PAIRS])
    dK = [_sym([_d(adm[:, 10 + q], a, h) for q in range(6)]) for a in R3]
    DK = [[[dK[a][b][c] - sum(Gu[d][a][b] * K[d][c] + Gu[d][a][c] * K[b][d] for d in R3)
            for c in R3] for b in R3] for a in R3]
    return I, g, gu, R, K, DK, dgt, gt


def _constraints(u, adm, p, h):
    I, g, gu, R, K, DK, dgt, gt = _curvature(u, adm, p, h)
    Rs = sum(gu[a][b] * R[a][b] for a in R3 for b in R3)
    Kud = [[sum(gu[a][c] * K[c][b] for c in R3) for b in R3] for a in R3]
    tr = Kud[0][0] + Kud[1][1] + Kud[2][2]
    H = Rs + tr * tr - sum(Kud[a][b] * Kud[b][a] for a in R3 for b in R3)
    Md = [sum(gu[b][c] * (DK[c][b][a] - DK[a][b][c]) for b in R3 for c in R3) for a in R3]
    M = sum(gu[a][b] * Md[a] * Md[b] for a in R3 for b in R3)
    gtu = _inv(gt)
    Gc = _christoffel(dgt, gtu)[1]
    Zu = [I[14 + a] - sum(gtu[b][c] * Gc[a][b][c] for b in R3 for c in R3) for a in R3]
    Zs = 0.25 * sum(g[a][b] * Zu[a] * Zu[b] for a in R3 for b in R3)
    C = H * H + M + I[17] ** 2 + 4 * Zs
    return _pad(torch.stack([C, H, M, Zs] + Md, 1))


def _norms(u, con, h):
    s = lambda f: _crop(f, (4, 4, 4))[:, :-1, :-1, :-1].sum() * h[0] * h[1] * h[2]  # noqa: E731
    return torch.stack([s(con[:, 1] ** 2), s(con[:, 2].abs())] + [s(con[:, 4 + a] ** 2) for a in R3]
                       + [s(con[:, 3].abs()), s(u[:, 17] ** 2), s(con[:, 0].abs())])


def _psi4(case, mesh, u, adm, p, h):
    _, g, gu, R, K, DK, _, _ = _curvature(u, adm, p, h)
    Rs = sum(gu[a][b] * R[a][b] for a in R3 for b in R3)
    tr = sum(gu[a][b] * K[a][b] for a in R3 for b in R3)
    x, y, z = [_crop(c.expand(mesh.nblocks, *reversed(mesh.nn)), (4, 4, 4))
               for c in _coords(case, mesh)]
    x = torch.where(x * x + y * y < 1e-10, x + 1e-8, x)
    dot = lambda l, r: sum(g[a][b] * l[a] * r[b] for a in R3 for b in R3)  # noqa: E731
    unit = lambda l: [c / dot(l, l).sqrt() for c in l]  # noqa: E731
    off = lambda l, *n: [l[a] - sum(dot(m, l) * m[a] for m in n) for a in R3]  # noqa: E731
    wv = unit([-y, x, torch.zeros_like(x)])
    uv = unit(off([x, y, z], wv))
    vv = unit(off([x * z, y * z, -x * x - y * y], wv, uv))
    re = im = 0
    for a in R3:
        for b in R3:
            T = (vv[a] * vv[b] - wv[a] * wv[b], -vv[a] * wv[b] - wv[a] * vv[b])
            s = -0.25 * (R[a][b] + tr * K[a][b] - sum(
                gu[c][d] * K[a][c] * K[d][b] for c in R3 for d in R3))
            for c in R3:
                s = s - 0.5 * (DK[b][a][c] - DK[c][a][b]) * uv[c]
                for d in R3:
                    s = s - 0.25 * uv[d] * uv[c] * (
                        g[d][c] * R[a][b] + g[a][b] * R[d][c] - g[d][b] * R[a][c]
                        - g[a][c] * R[d][b] - 0.5 * Rs * (g[d][c] * g[a][b] - g[d][b] * g[a][c])
                        + K[d][c] * K[a][b] - K[d][b] * K[a][c])
            re, im = re + s * T[0], im + s * T[1]
    return _fill(_pad(torch.stack([re, im], 1)), mesh)


class _P:
    """The options _rhs reads, with the package's defaults."""

    def __init__(self, **kw):
        self.__dict__ = dict(dict(
            chi_div_floor=-1000.0, diss=0.0, eps_floor=1e-12, damp_kappa1=0.0, damp_kappa2=0.0,
            lapse_oplog=2.0, lapse_harmonicf=1.0, lapse_harmonic=0.0, lapse_advect=1.0,
            lapse_K=0.0, shift_Gamma=1.0, shift_advect=1.0, shift_eta=2.0), **kw)


def _finalize(u, mesh, p):
    """The ghosts of a loaded state: fill, then the algebraic constraints on
    the ghosts only."""
    f = _fill(u, mesh)
    c = _alg_constr(f, p.eps_floor)
    c[..., 4:-4, 4:-4, 4:-4] = f[..., 4:-4, 4:-4, 4:-4]
    return c


def exact(case, seed):
    kind = case["kind"]
    if kind == "refined":
        # the multilevel prolongation's lists of message boxes have no short
        # form: checked against the start's outputs only
        return None
    mesh, p = _mesh(case), _P(**_params(case))
    h = [(mesh.xmax[a] - mesh.xmin[a]) / (mesh.nb[a] * mesh.nx[a]) for a in R3]
    dt = 0.25 * min(h)
    if kind == "initial":
        data = _adm_data(case, mesh, seed)
        u = _finalize(_alg_constr(_adm_to_z4c(data, h), p.eps_floor), mesh, p)
        adm = _z4c_to_adm(u)
        adm[..., 4:-4, 4:-4, 4:-4] = data[..., 4:-4, 4:-4, 4:-4]
        return {"u": u, "adm": adm}
    if kind == "jobs":
        out = {"norms": []}
        for j in range(case["jobs"]):
            u = _finalize(_state(case, mesh, seed, j), mesh, p)
            for _ in range(case["steps"]):
                u = _step(u, p, h, mesh, dt)
            out["norms"].append(_norms(u, _constraints(u, _z4c_to_adm(u), p, h), h))
            out[f"u{j}"] = u
        out["norms"] = torch.stack(out["norms"])
        return out
    u = _finalize(_state(case, mesh, seed), mesh, p)
    if kind == "rhs":
        return {"rhs": _pad(_rhs(u, p, h))}
    if kind == "evolve":
        som = _sommerfeld(case, mesh, h) if case["bc"] == "sommerfeld" else None
        for _ in range(case["steps"]):
            u = _step(u, p, h, mesh, dt, case["integ"], som)
        out = {"u": u, "adm": _z4c_to_adm(u)}
        if case["con"]:
            out["con"] = _constraints(u, out["adm"], p, h)
        return out
    if kind == "diagnostics":
        adm = _z4c_to_adm(u)
        con = _constraints(u, adm, p, h)
        return {"norms": _norms(u, con, h), "adm": adm, "con": con}
    if kind == "psi4":
        # the multipoles need the geodesic spheres' tables
        return {"weyl": _psi4(case, mesh, u, _z4c_to_adm(u), p, h), "inner": None, "outer": None}
    from torch.utils.checkpoint import checkpoint
    u.requires_grad_(True)
    v = _step(u, p, h, mesh, dt,
              stage_wrap=lambda f, *x: checkpoint(f, *x, use_reentrant=False))
    return {"ubar": torch.autograd.grad(v, u, _cotangent(tuple(v.shape), seed))[0]}
