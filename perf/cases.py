"""The work that users of the framework have it do, as cases with their inputs, one pass and its result.

Most passes are time steps: a driver holds a state on the device, hands it to the solver, has one step of it done
(imex_step) and takes the new state back, so that every pass does the same work.  Beside them stand the parts a driver
can call by itself (the explicit half of a stage, a magnetic solve, a pressure solve), the ensemble and the adjoint.

`listed()` names the cases, `draw(rng)` gives others of the same ranges, `prepare(case, seed)` makes what a program
has in hand before the call, `run(state)` is one pass, `work(case)` its compulsory traffic, and `exact(case, seed)`
the 64-bit result of the single parts.  Whole steps, the ensemble and the adjoint have none: their implicit solves stop
at a tolerance, and restating the whole scheme here would only repeat the oracle.
"""
import ctypes
import math

import numpy as np
import torch

import imex_b200 as ix
from imex_b200 import problems

# The settings of the benchmark's workloads (bench.py) and of the reference's Orszag-Tang test.
SHEET = dict(recon="WENO5", magfield="PotentialA", floor_on=1, p_floor=1e-8, theta=0.5, GMREStol=1e-14)
VORTEX = dict(recon="VanLeer", magfield="StaggerCT", GMREStol=1e-12)
RANDOM = dict(recon="Minmod", magfield="StaggerCT", floor_on=1)
BLAST = dict(recon="WENO5", magfield="StaggerCT", floor_on=1, p_floor=1e-8, theta=0.5, GMREStol=1e-14)
ENERGY = dict(recon="Minmod", magfield="StaggerCT", formula="EnergyFormula")


def listed():
    return [
        # the smallest run of the benchmark: launches and barriers
        dict(name="step_vortex_64", kind="vortex", nx=64, ny=64, rks=2, precision="fp64"),
        # a sheet of odd sides, as a resolution study has
        dict(name="step_sheet_251x173", kind="sheet", nx=251, ny=173, rks=3, precision="fp64"),
        # the headline: 1024^2 vortex sheet, WENO5, A form, pressure floor, RK3
        dict(name="step_sheet_1024", kind="sheet", nx=1024, ny=1024, rks=3, precision="fp64"),
        # the largest: planes far beyond the L2
        dict(name="step_sheet_2048", kind="sheet", nx=2048, ny=2048, rks=3, precision="fp64"),
        # the stiff field: Redlich-Kwong gas, beta 0.1, many Krylov steps; plain and in the mixed form its workload asks for
        dict(name="step_random_768", kind="random", nx=768, ny=768, rks=2, precision="fp64"),
        dict(name="step_random_1024_mixed", kind="random", nx=1024, ny=1024, rks=2, precision="mixed"),
        # an open domain, ragged tiles, B form
        dict(name="step_blast_700x450", kind="blast", nx=700, ny=450, rks=3, precision="fp64"),
        # the energy formula on the reference's Orszag-Tang test
        dict(name="step_energy_320", kind="energy", nx=320, ny=320, rks=2, precision="fp64"),
        # an ensemble of independent runs on uneven grids, mixed form
        dict(name="ensemble_20", kind="ensemble", members=20, smin=64, smax=256, rks=2, precision="mixed"),
        # backward: the vector-Jacobian product of three steps
        dict(name="adjoint_128", kind="adjoint", nx=128, ny=128, rks=2, steps=3),
        # the explicit half of a stage on its own: reconstruction and both face fluxes
        dict(name="explicit_1000x700", kind="explicit", nx=1000, ny=700, recon="WENO5"),
        # one pressure solve with the floor on, device vectors
        dict(name="pressure_513x400", kind="pressure", nx=513, ny=400),
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["vortex", "sheet", "sheet", "random", "blast", "energy", "ensemble", "adjoint", "explicit", "pressure"])
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(4, 20), smin=48, smax=side(96, 256), rks=2, precision=rng.choice(["fp64", "mixed"]))
    if kind == "adjoint":
        n = side(48, 160)
        return dict(kind=kind, nx=n, ny=n, rks=2, steps=rng.randint(1, 3))
    if kind == "random":
        n = side(96, 768)
        return dict(kind=kind, nx=n, ny=n, rks=2, precision=rng.choice(["fp64", "mixed"]))
    longest = 1000 if kind in ("blast", "energy") else 1600
    nx, ny = side(48, longest), side(48, longest)
    if kind == "explicit":
        return dict(kind=kind, nx=nx, ny=ny, recon=rng.choice(["WENO5", "VanLeer", "Minmod"]))
    if kind == "pressure":
        return dict(kind=kind, nx=nx, ny=ny)
    return dict(kind=kind, nx=nx, ny=ny, rks=rng.choice([2, 3]), precision=rng.choice(["fp64", "fp64", "mixed"]))


# ------------------------------------------------------------------ inputs
def _vary(p, seed):
    """The problem with smooth seeded changes of velocity and pressure (B and A stay, so div B = 0 stays)."""
    rng = np.random.default_rng(seed)
    x = (2.0 * math.pi / p.nx) * (np.arange(p.nx) + 0.5)
    y = (2.0 * math.pi / p.ny) * (np.arange(p.ny) + 0.5)
    size = 0.05 * max(float(np.sqrt(p.prim[1] ** 2 + p.prim[2] ** 2).max()), 1e-6)
    for k in (1, 2):
        a, b = rng.uniform(0.0, 2.0 * math.pi, 2)
        p.prim[k] += size * np.cos(y + a)[:, None] * np.sin(2.0 * x + b)[None, :]
    a, b = rng.uniform(0.0, 2.0 * math.pi, 2)
    p.prim[4] *= 1.0 + 0.05 * np.sin(2.0 * y + a)[:, None] * np.cos(x + b)[None, :]
    return p


def _problem(case, seed):
    """(problem, settings) of a whole-step case."""
    kind, nx, ny = case["kind"], case["nx"], case["ny"]
    if kind == "vortex":
        return _vary(problems.vortex(nx, ny), seed), dict(VORTEX)
    if kind == "sheet":
        return _vary(problems.vortex_sheet(nx, ny), seed), dict(SHEET)
    if kind == "blast":
        return _vary(problems.open_blast(nx, ny), seed), dict(BLAST)
    if kind == "energy":
        return _vary(problems.reference_test("Orszag_Tang", nx, ny), seed), dict(ENERGY, time_stop=1e30)
    # the low-Mach field starts far below its magnetic speeds and its step grows from the explicit limit; a run's
    # steps settle at two to five times that limit, so the step is set to three times it
    p = problems.random_field(nx, seed=seed)
    fast = math.sqrt(float((p.prim[5] ** 2 + p.prim[6] ** 2).max()) + 3.0)
    return p, dict(RANDOM, fixed_dt=3 * 0.4 * p.dx / fast)


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _ptr(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def _ok(sv, rc):
    sv._check(rc)


def _new_state(n):
    return [torch.empty(k * n, dtype=torch.float64, device="cuda") for k in (8, 1, 1, 3)]


def _take(sv, out):
    sv.download_state_ptr(*[t.data_ptr() for t in out])


def _gas(nx, ny, seed):
    """A smooth conserved state (8 planes) and two like it on the unit square, as stage buffers hold them."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = (torch.arange(nx, dtype=torch.float64, device="cuda") + 0.5) * (2 * math.pi / nx)
    y = (torch.arange(ny, dtype=torch.float64, device="cuda") + 0.5) * (2 * math.pi / ny)

    def wave(size):
        f = torch.zeros(ny, nx, dtype=torch.float64, device="cuda")
        r = torch.rand(4, 3, generator=g, device="cuda", dtype=torch.float64).tolist()
        for m, (a, b, c) in enumerate(r):
            f += size * (c - 0.5) * torch.cos((m % 3 + 1) * y + 6.283 * a)[:, None] * torch.sin((m // 2 + 1) * x + 6.283 * b)[None, :]
        return f

    def state():
        rho = 1.0 + 0.2 * wave(1.0)
        v = [wave(0.8) for _ in range(3)]
        B = [wave(0.7) for _ in range(3)]
        p = 1.0 + 0.3 * wave(1.0)
        p = torch.where((x > 2.0)[None, :] & (y > 3.0)[:, None], 0.4 * p, p)  # a jump, for the limiters
        E = 1.5 * p + 0.5 * rho * sum(c * c for c in v) + 0.5 * sum(c * c for c in B)
        return torch.stack([rho, *[rho * c for c in v], E, *B])

    first = state()
    return first, first + 1e-2 * (state() - first), first + 1e-2 * (state() - first)


def _part_solver(case, settings):
    sv = ix.Solver(case["nx"], case["ny"], dict(settings, vortex_test=0), (0.0, 1.0, 0.0, case["ny"] / case["nx"]), 2)
    return sv


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        # the grids are the case's, not the seed's: only the vortices differ
        grids = problems.vortex_ensemble(case["members"], 7, case["smin"], case["smax"])
        rng = np.random.default_rng(seed)
        ps = [problems.vortex(g.nx, kappa=rng.uniform(0.5, 1.5), mu=rng.uniform(0.5, 1.5)) for g in grids]
        b = ix.Batch(ps, case["rks"], dict(VORTEX, precision=case["precision"]))
        b.step(3)
        sizes = [13 * p.nx * p.ny for p in ps]
        flat = torch.empty(sum(sizes), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        return dict(kind=kind, batch=b, flat=flat)
    if kind == "adjoint":
        p = problems.perturbed_vortex(case["nx"], seed=seed, modes=8).problem()
        sv = ix.Solver.for_problem(p, case["rks"], dict(VORTEX, fixed_dt=0.1 * p.dx))
        start = [_dev(p.prim), _dev(p.bx), _dev(p.by), _dev(p.A)]
        rng = np.random.default_rng(seed)
        lam = rng.standard_normal((8, p.ny, p.nx))
        torch.cuda.synchronize()
        return dict(kind=kind, sv=sv, start=start, lam=lam, steps=case["steps"])
    if kind == "explicit":
        sv = _part_solver(case, dict(SHEET, recon=case["recon"]))
        Qe, Qs, u = _gas(case["nx"], case["ny"], seed)
        torch.cuda.synchronize()
        for buf, t in (("Qe", Qe), ("Qs", Qs), ("cons", u)):
            _ok(sv, sv.lib.imex_set_buffer(sv.ctx, ix.BUF[buf], 0, _ptr(t)))
        sv.set_scalars(a_max=1.3)
        out = [torch.empty(8, case["ny"], case["nx"], dtype=torch.float64, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()
        return dict(kind=kind, sv=sv, h=0.2 / case["nx"], out=out)
    if kind == "pressure":
        sv = _part_solver(case, SHEET)
        Qe, Qs, u = _gas(case["nx"], case["ny"], seed)
        torch.cuda.synchronize()
        for buf, t in (("Qe", Qe), ("Qs", Qs), ("cons", u)):
            _ok(sv, sv.lib.imex_set_buffer(sv.ctx, ix.BUF[buf], 0, _ptr(t)))
        sv.set_scalars(vx_max=0.9, vy_max=0.7)
        stream = torch.cuda.Stream()
        sv.set_stream(stream.cuda_stream)
        b = _pressure_rhs(Qe)
        p0 = b / 1.5
        torch.cuda.synchronize()
        return dict(kind=kind, sv=sv, h=0.8 / case["nx"], b=b, p0=p0, p=torch.empty_like(p0), stream=stream)
    p, settings = _problem(case, seed)
    sv = ix.Solver.for_problem(p, case["rks"], dict(settings, precision=case["precision"]))
    for _ in range(3):  # past the first steps, whose dt is still growing
        sv.step()
    start, out = _new_state(sv.N), _new_state(sv.N)
    torch.cuda.synchronize()
    _take(sv, start)
    lines = None
    if kind == "blast":  # the boundary normal faces belong to the state too
        lines = [_dev(a) for a in sv.boundary_faces()]
    torch.cuda.synchronize()
    return dict(kind=kind, sv=sv, start=start, out=out, lines=lines)


def run(state):
    kind = state["kind"]
    if kind == "ensemble":
        b, flat = state["batch"], state["flat"]
        b.step(1)
        at = flat.data_ptr()
        for sv in b.members:
            n = 8 * sv.N
            sv.download_state_ptr(at, at + 8 * n, at + 9 * n, at + 10 * n)
            at += 13 * n
        return flat
    sv = state["sv"]
    if kind == "adjoint":
        sv.upload_state_ptr(*[t.data_ptr() for t in state["start"]])
        return sv.adjoint_vjp(state["steps"], state["lam"], checkpoint_every=2)
    if kind == "explicit":
        first, second = state["out"]
        sv.TVDReconstruction()
        sv.RusanovC_Update(state["h"])
        _ok(sv, sv.lib.imex_get_buffer(sv.ctx, ix.BUF["cons"], 0, _ptr(first)))
        sv.Pressure_flux_Update(state["h"])
        _ok(sv, sv.lib.imex_get_buffer(sv.ctx, ix.BUF["cons"], 0, _ptr(second)))
        return [first, second]
    if kind == "pressure":
        with torch.cuda.stream(state["stream"]):
            state["p"].copy_(state["p0"])
        sv.prepare_operator("pressure_L", state["h"])
        _ok(sv, sv.lib.imex_pressure_nested_newton(sv.ctx, _ptr(state["p"]), _ptr(state["b"]), None))
        return state["p"]
    sv.upload_state_ptr(*[t.data_ptr() for t in state["start"]])
    if state["lines"] is not None:
        _ok(sv, sv.lib.imex_set_boundary_faces(sv.ctx, *[_ptr(t) for t in state["lines"]]))
    sv.step()
    _take(sv, state["out"])
    return state["out"]


def work(case):
    """Compulsory traffic in bytes: a step reads and writes 13 planes; flops as rough counts per cell."""
    kind = case["kind"]
    if kind == "ensemble":
        cells = sum(p.nx * p.ny for p in problems.vortex_ensemble(case["members"], 7, case["smin"], case["smax"]))
        return {"bytes": 8.0 * 26 * cells, "flops": 2000.0 * case["rks"] * cells}
    cells = case["nx"] * case["ny"]
    if kind == "adjoint":  # the state and the cotangent in, ten planes of gradient out
        return {"bytes": 8.0 * 31 * cells, "flops": 8000.0 * case["rks"] * case["steps"] * cells}
    if kind == "explicit":  # Qe, Qs (5 planes) and B in, twice 5 planes out
        return {"bytes": 8.0 * (5 + 5 + 3 + 5 + 5) * cells, "flops": 700.0 * cells}
    if kind == "pressure":  # b, p0, and rho, momentum, E, B of Qe in, p out
        return {"bytes": 8.0 * (2 + 8 + 1 + 1) * cells, "flops": 400.0 * cells}
    return {"bytes": 8.0 * 26 * cells, "flops": 2000.0 * case["rks"] * cells}


# ------------------------------------------------------------------ 64-bit results of the single parts
def _at(a, di, dj):
    """a at (i + di, j + dj), periodic."""
    return torch.roll(a, (-dj, -di), (-2, -1))


def _face_values(a, scheme, step):
    """Left and right face value of each cell of plane a along the direction of `step` (di, dj)."""
    s = lambda m: _at(a, m * step[0], m * step[1])  # noqa: E731
    um2, um1, u0, up1, up2 = s(-2), s(-1), a, s(1), s(2)
    sL, sR = u0 - um1, up1 - u0
    if scheme == "Minmod":
        c = torch.where(sL * sR <= 0, torch.zeros_like(sL), torch.where(sR.abs() <= sL.abs(), sR, sL))
        return u0 - 0.5 * c, u0 + 0.5 * c
    if scheme == "VanLeer":
        small = sR.abs() < 1e-16
        r = sL / torch.where(small, torch.ones_like(sR), sR)
        c = torch.where(small | (r < 0), torch.zeros_like(r), torch.minimum(2 / (1 + r), 2 * r / (1 + r)))
        return u0 - 0.5 * c * sL, u0 + 0.5 * c * sR
    beta = [(13 / 12 * (um2 - 2 * um1 + u0) ** 2 + 0.25 * (um2 - 4 * um1 + 3 * u0) ** 2 + 1e-6) ** 2,
            (13 / 12 * (um1 - 2 * u0 + up1) ** 2 + 0.25 * (um1 - up1) ** 2 + 1e-6) ** 2,
            (13 / 12 * (u0 - 2 * up1 + up2) ** 2 + 0.25 * (3 * u0 - 4 * up1 + up2) ** 2 + 1e-6) ** 2]

    def mix(d, q):
        w = [d[k] / beta[k] for k in range(3)]
        return sum(w[k] * q[k] for k in range(3)) / sum(w)

    left = mix((0.3, 0.6, 0.1), ((-um2 + 5 * um1 + 2 * u0) / 6, (2 * um1 + 5 * u0 - up1) / 6, (11 * u0 - 7 * up1 + 2 * up2) / 6))
    right = mix((0.1, 0.6, 0.3), ((2 * um2 - 7 * um1 + 11 * u0) / 6, (-um1 + 5 * u0 + 2 * up1) / 6, (2 * u0 + 5 * up1 - up2) / 6))
    return left, right


def _flux(q, d, magnetic):
    v = [q[k] / q[0] for k in (1, 2, 3)]
    f = [q[1 + d], q[1] * v[d], q[2] * v[d], q[3] * v[d], 0.5 * q[0] * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2) * v[d]]
    if magnetic:
        B = q[5:8]
        B2, vB = (B * B).sum(0), v[0] * B[0] + v[1] * B[1] + v[2] * B[2]
        for k in range(3):
            f[1 + k] = f[1 + k] - B[d] * B[k] + (0.5 * B2 if k == d else 0.0)
        f[4] = f[4] + v[d] * B2 - B[d] * vB
    return torch.stack(f)


def _exact_explicit(case, seed):
    Qe, Qs, u = _gas(case["nx"], case["ny"], seed)
    dx = 1.0 / case["nx"]
    h, a_max, out = 0.2 / case["nx"], 1.3, []
    lows, highs = {}, {}
    for d, step in ((0, (1, 0)), (1, (0, 1))):
        both = [_face_values(Qe[k], case["recon"], step) for k in range(5)]
        lows[d], highs[d] = torch.stack([b[0] for b in both]), torch.stack([b[1] for b in both])
    for magnetic in (False, True):
        new = Qs[:5].clone()
        for d, step in ((0, (1, 0)), (1, (0, 1))):
            qL = torch.cat([highs[d], u[5:8]])  # the state left of the face i + 1/2
            qR = torch.cat([_at(lows[d], *step), _at(u[5:8], *step)])
            F = 0.5 * (_flux(qL, d, magnetic) + _flux(qR, d, magnetic)) - 0.5 * a_max * (qR[:5] - qL[:5])
            new = new - h / dx * (F - _at(F, -step[0], -step[1]))
        out.append(torch.cat([new, u[5:8]]))
    return out


def _pressure_rhs(Qe):
    """A right-hand side like a stage's: 1.5 p of the explicit state with a small ripple."""
    m2, B2 = (Qe[1:4] ** 2).sum(0), (Qe[5:8] ** 2).sum(0)
    e = Qe[4] - 0.5 * m2 / Qe[0] - 0.5 * B2
    return (e * (1.0 + 0.02 * torch.sin(7.0 * Qe[1]))).contiguous()


def _shock(Q, dx, dy, gamma, kappa):
    v = Q[1:4] / Q[0]
    B2 = (Q[5:8] ** 2).sum(0)
    p = (gamma - 1) * (Q[4] - 0.5 * Q[0] * (v * v).sum(0) - 0.5 * B2)
    c = torch.sqrt((gamma * p + B2) / Q[0])
    near = lambda a: torch.stack([_at(a, i, j) for i in (-1, 0, 1) for j in (-1, 0, 1)])  # noqa: E731
    low = near(c).amin(0)
    div = (_at(v[0], 1, 0) - _at(v[0], -1, 0)) / (2 * dx) + (_at(v[1], 0, 1) - _at(v[1], 0, -1)) / (2 * dy)
    chi = (-(min(dx, dy) * div + kappa * low) / (kappa * low)).clamp(0.0, 1.0)
    return near(chi).amax(0)


def _exact_pressure(case, seed):
    Qe, Qs, u = _gas(case["nx"], case["ny"], seed)
    gamma, dx = 5.0 / 3.0, 1.0 / case["nx"]
    dy, h = dx, 0.8 / case["nx"]
    v = Qe[1:4] / Qe[0]
    e = Qe[4] / Qe[0] - 0.5 * (v * v).sum(0) - 0.5 * (Qe[5:8] ** 2).sum(0) / Qe[0]
    hh = gamma * e * Qe[0] / u[0]
    eta = _shock(Qe, dx, dy, gamma, 0.001)
    nu = (0.9 * dx, 0.7 * dy)
    a = 1.0 / (gamma - 1.0)

    def L(p):
        out = a * p
        for d, step in ((0, (1, 0)), (1, (0, 1))):
            w = dx if d == 0 else dy
            grad = _at(p, *step) - p
            f = 0.5 * (hh + _at(hh, *step)) * grad
            g = 0.5 * (eta + _at(eta, *step)) * grad * nu[d] * a * h
            out = out - (h * h * (f - _at(f, -step[0], -step[1])) + g - _at(g, -step[0], -step[1])) / (w * w)
        return out

    b = _pressure_rhs(Qe)
    diag = a + h * h * sum((2 * hh + _at(hh, i, j) + _at(hh, -i, -j)) / 2 for i, j in ((1, 0), (0, 1))) / (dx * dx)
    return _solve(L, b, b * (gamma - 1.0), diag)


def _solve(A, b, x, diag, restart=40, cycles=12):
    """Restarted GMRES, left-preconditioned by diag, until the residual stops falling."""
    last = math.inf
    for _ in range(cycles):
        r = (b - A(x)) / diag
        norm = float(r.norm())
        if norm == 0.0 or norm > 0.5 * last:
            break
        last = norm
        V = [(r / norm).reshape(-1)]
        H = torch.zeros(restart + 1, restart, dtype=torch.float64)
        for j in range(restart):
            w = (A(V[j].reshape(b.shape)) / diag).reshape(-1)
            for _twice in range(2):
                for i in range(j + 1):
                    c = torch.dot(V[i], w)
                    H[i, j] += float(c)
                    w = w - c * V[i]
            H[j + 1, j] = float(w.norm())
            if H[j + 1, j] < 1e-17:
                break
            V.append(w / H[j + 1, j].item())
        k = len(V) - 1
        rhs = torch.zeros(k + 1, dtype=torch.float64)
        rhs[0] = norm
        y = torch.linalg.lstsq(H[: k + 1, :k], rhs).solution
        x = x + sum(float(y[i]) * V[i] for i in range(k)).reshape(b.shape)
    return x


def exact(case, seed):
    if case["kind"] == "explicit":
        return _exact_explicit(case, seed)
    if case["kind"] == "pressure":
        return _exact_pressure(case, seed)
    return None
