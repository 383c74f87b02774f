"""The solves of the row-marching kernels (imex_b200/csrc/march_solve.cuh) at the sizes where
their cut of the grid can go wrong: grids narrower than a strip (62 columns of a one-component
vector, 30 and 28 of the B and A forms), one column past it, runs cut short at the last row, and
enough tasks for several blocks; periodic and transmissive; FP64 and mixed; conjugate gradients
and GMRES through their slot limits.

Each solve's right-hand side is the operator (imex_apply_operator, which test_gpu_parity.py pins
to the oracle) applied to a known vector of size one.  The error of the solution is the stopping
tolerance, 1e-13 relative plus 1e-13 absolute in the preconditioned residual, times the
condition number, below 1e3 for these steps (the diagonals lie between 1 and about 30): 1e-10 with
the vector's norm.  The mixed form stops at mixed_outer_tol = 1e-10: 1e-7."""
from __future__ import annotations

import numpy as np
import pytest

import imex_b200 as ix
from conftest import rel
from imex_b200.problems import open_blast, random_field, vortex, vortex_sheet

pytestmark = pytest.mark.gpu

SIZES = [(4, 4), (5, 9), (28, 7), (29, 4), (30, 6), (31, 5), (61, 8), (62, 5), (63, 4), (125, 7), (4, 131), (130, 71)]
B_FORM = dict(recon="VanLeer", magfield="StaggerCT", GMREStol=1e-13)
A_FORM = dict(recon="WENO5", magfield="PotentialA", GMREStol=1e-13)
ENERGY = dict(recon="Minmod", magfield="StaggerCT", formula="EnergyFormula", GMREStol=1e-13)
OPS = [("pressure_L", B_FORM, "vortex"), ("pressure_J", B_FORM, "vortex"), ("magnetic_B", B_FORM, "vortex"),
       ("magnetic_A", A_FORM, "sheet"), ("energy", ENERGY, "vortex"), ("pressure_L", B_FORM, "blast"),
       ("magnetic_B", B_FORM, "blast"), ("energy", ENERGY, "blast")]


def _solver(kind, nx, ny, settings):
    prob = {"vortex": vortex, "sheet": vortex_sheet, "blast": open_blast}[kind](nx, ny)
    sv = ix.Solver.for_problem(prob, 2, settings)
    for name in ("Qe", "Qs"):  # stage buffers of a state with variation in every plane
        sv.set_buffer(name, sv.cons())
    sv.set_scalars(vx_max=0.8, vy_max=0.9, B_max_x=0.7, B_max_y=0.6)
    return sv, prob


def _known(sv, op, seed=3):
    n = sv.nx * sv.ny * (3 if op.startswith("magnetic") else 1)
    return np.random.default_rng(seed).standard_normal(n)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("op,settings,kind", OPS)
def test_march_solves_recover_a_known_vector(op, settings, kind, precision):
    for nx, ny in SIZES:
        sv, prob = _solver(kind, nx, ny, dict(settings, precision=precision, mixed_solves=7))
        sv.prepare_operator(op, 2.0 * min(prob.dx, prob.dy))
        if op == "pressure_J":  # some floored cells, whose slope is Mbig
            sv.set_newton_state(np.where(np.arange(sv.N) % 7 == 3, -1.0, 1.0), 50.0)
        x = _known(sv, op)
        got, st = sv.gmres(op, np.zeros_like(x), sv.apply_operator(op, x))
        assert st["status"] == 0
        assert rel(got, x) <= (1e-10 if precision == "fp64" else 1e-7), (nx, ny, rel(got, x))
        sv.close()


@pytest.mark.parametrize("restart", [1, 2, 3, 25, 30])
@pytest.mark.parametrize("op,settings,kind", [OPS[0], OPS[2], OPS[3], OPS[4]])
def test_march_solves_with_few_and_many_slots(op, settings, kind, restart):
    """Restarted GMRES, and conjugate gradients that fill their residual slots many times."""
    sv, prob = _solver(kind, 63, 41, dict(settings, gmres_restart=restart))
    sv.prepare_operator(op, 2.0 * min(prob.dx, prob.dy))
    x = _known(sv, op)
    got, st = sv.gmres(op, np.zeros_like(x), sv.apply_operator(op, x))
    assert st["status"] == 0 and rel(got, x) <= 1e-10, (st, rel(got, x))
    sv.close()


@pytest.mark.parametrize("nx,ny", [(5, 9), (63, 4), (130, 71)])
@pytest.mark.parametrize("eos", ["IDEAL_GAS", "REDLICH_KWONG"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_march_newton_matches_the_tile_kernels(nx, ny, eos, precision):
    """The nested Newton against the exact arithmetic's (the tile kernels) on a right-hand side
    that floors some cells.  Both stop at a residual of 1e-8 of the first plus 1e-8; the Newton
    converges quadratically, so the iterates agree to about the square of that: 1e-9."""
    n = min(nx, ny)
    res = []
    for arith in ("exact", "fast"):
        sv = ix.Solver.for_problem(vortex(nx, ny), 2, dict(B_FORM, arith=arith, eos_type=eos, m_alfa=0.05, m_b=0.1,
                                                           p_floor=0.05, theta=0.5, precision=precision))
        for name in ("Qe", "Qs"):
            sv.set_buffer(name, sv.cons())
        sv.set_scalars(vx_max=0.8, vy_max=0.9)
        sv.prepare_operator("pressure_L", 0.5 * min(10.0 / nx, 10.0 / ny))
        b = 1.5 * np.ones(sv.N)
        b[:: 11] = 0.02
        p, st = sv.nested_newton(np.full(sv.N, 0.9), b)
        assert st["newton_iters"] >= 1
        res.append(p)
        sv.close()
    assert rel(res[1], res[0]) <= 1e-9, (n, rel(res[1], res[0]))


@pytest.mark.parametrize("nx,ny,kind", [(1201, 601, "vortex"), (700, 1100, "blast")])
@pytest.mark.parametrize("floors", [False, True])
@pytest.mark.parametrize("precision,restart", [("fp64", 30), ("fp64", 12), ("fp64", 3), ("mixed", 30)])
def test_march_newton_of_long_tasks(nx, ny, kind, floors, precision, restart):
    """Tasks of eight rows and more (some short at the last row), whose residual passes copy their
    rows ahead: with few and many vectors in the pending update, with cells floored after the
    first iterate.  Tolerance as above."""
    res = []
    prob = {"vortex": vortex, "blast": open_blast}[kind](nx, ny)
    for arith in ("exact", "fast"):
        sv = ix.Solver.for_problem(prob, 2, dict(B_FORM, arith=arith, p_floor=0.05, theta=0.5, precision=precision,
                                                 gmres_restart=restart))
        for name in ("Qe", "Qs"):
            sv.set_buffer(name, sv.cons())
        sv.set_scalars(vx_max=0.8, vy_max=0.9)
        sv.prepare_operator("pressure_L", 2.0 * min(prob.dx, prob.dy))
        b = 1.5 + 0.3 * np.sin(0.05 * np.arange(sv.N))
        if floors:
            b[::11] = 0.02
        p, st = sv.nested_newton(np.full(sv.N, 0.9), b)
        assert st["newton_iters"] >= 1
        res.append(p)
        sv.close()
    assert rel(res[1], res[0]) <= 1e-9, rel(res[1], res[0])


def test_march_falls_back_where_conjugate_gradients_break_down():
    """A negative face weight (an operator that is not positive definite) hands the solve to GMRES."""
    sv, prob = _solver("vortex", 63, 41, B_FORM)
    sv.prepare_operator("pressure_J", 2.0 * min(prob.dx, prob.dy))
    sv.set_newton_state(np.where(np.arange(sv.N) % 5 == 2, -1.0, 1.0), -40.0)  # slopes of both signs
    x = _known(sv, "pressure_J")
    got, st = sv.gmres("pressure_J", np.zeros_like(x), sv.apply_operator("pressure_J", x))
    assert st["status"] == 0 and rel(got, x) <= 1e-8, (st, rel(got, x))
    sv.close()


def test_march_newton_is_bit_reproducible():
    runs = []
    for _ in range(2):
        sv = ix.Solver.for_problem(random_field(65), 2, dict(recon="Minmod", magfield="StaggerCT", precision="mixed"))
        for _ in range(2):
            sv.step()
        runs.append(sv.cons())
        sv.close()
    np.testing.assert_array_equal(runs[0], runs[1])


@pytest.mark.parametrize("restart", [1, 11, 12, 13, 30])
@pytest.mark.parametrize("nx,ny,kind", [(63, 41, "vortex"), (131, 90, "blast")])
def test_march_mixed_magnetic_solve_around_its_ring(nx, ny, kind, restart):
    """The mixed B-form solve holds twelve FP32 vectors in its ring: Krylov spaces below, at and past it.
    With one vector a sweep gains less than half, where the mixed form stops: there the iterate is the
    tile kernels' (the exact arithmetic), after four FP32 sweeps of error 6e-8 times a condition
    number below 1e3 each."""
    settings = dict(B_FORM, precision="mixed", mixed_solves=7, gmres_restart=restart, mixed_max_refine=400)
    sv, prob = _solver(kind, nx, ny, settings)
    sv.prepare_operator("magnetic_B", 6.0 * min(prob.dx, prob.dy))
    x = _known(sv, "magnetic_B")
    b = sv.apply_operator("magnetic_B", x)
    got, st = sv.gmres("magnetic_B", np.zeros_like(x), b)
    sv.close()
    assert st["status"] == 0
    if restart > 1:
        assert rel(got, x) <= 1e-7, (st, rel(got, x))
        return
    sv, prob = _solver(kind, nx, ny, dict(settings, arith="exact"))
    sv.prepare_operator("magnetic_B", 6.0 * min(prob.dx, prob.dy))
    want, st = sv.gmres("magnetic_B", np.zeros_like(x), b)
    sv.close()
    assert rel(got, want) <= 4 * 6e-8 * 1e3, rel(got, want)


def _newton_solver(nx, ny, steps, **settings):
    prob = vortex(nx, ny)
    sv = ix.Solver.for_problem(prob, 2, dict(B_FORM, **settings))
    for name in ("Qe", "Qs"):
        sv.set_buffer(name, sv.cons())
    sv.set_scalars(vx_max=0.8, vy_max=0.9)
    sv.prepare_operator("pressure_L", steps * min(prob.dx, prob.dy))
    return sv


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("floors", [False, True])
@pytest.mark.parametrize("nx,ny", [(63, 41), (700, 500)])
def test_newton_leaves_its_slopes_to_the_jacobian_operator(floors, nx, ny, precision):
    """IMEX_OP_PRESSURE_J after a nested Newton has the slopes of its last iterate (the reference's p_freeze),
    whatever was set before.  The operators agree to rounding: 1e-12."""
    out = []
    for arith in ("exact", "fast"):
        sv = _newton_solver(nx, ny, 0.1, arith=arith, p_floor=0.05, theta=0.5, precision=precision)
        sv.set_newton_state(np.where(np.arange(sv.N) % 3 == 1, -1.0, 1.0), 7.0)
        b = 1.5 * np.ones(sv.N)
        if floors:
            b[::11] = 0.002
        p, st = sv.nested_newton(np.full(sv.N, 0.9), b)
        assert st["status"] in (0, 7) and (p < 0.05).any() == floors
        out.append(sv.apply_operator("pressure_J", _known(sv, "pressure_J")))
        sv.close()
    assert rel(out[1], out[0]) <= 1e-12, rel(out[1], out[0])


def _indefinite(nx, ny, **settings):
    """pressure_J with slopes of both signs: not positive definite, so conjugate gradients break down."""
    sv, prob = _solver("vortex", nx, ny, dict(B_FORM, **settings))
    sv.prepare_operator("pressure_J", 2.0 * min(prob.dx, prob.dy))
    sv.set_newton_state(np.where(np.arange(sv.N) % 5 == 2, -1.0, 1.0), -40.0)
    return sv


def test_breakdown_leaves_gmres_its_restarts():
    """Twenty unknowns, one GMRES cycle of thirty: the cycle that the exact arithmetic solves the system in
    is still there after conjugate gradients broke down.  Tolerance as above."""
    sv = _indefinite(5, 4, gmres_max_restarts=1, gmres_restart=30)
    x = _known(sv, "pressure_J")
    got, st = sv.gmres("pressure_J", np.zeros_like(x), sv.apply_operator("pressure_J", x))
    assert st["status"] == 0 and rel(got, x) <= 1e-8, (st, rel(got, x))
    sv.close()


def test_breakdown_leaves_the_mixed_form_its_sweeps():
    """The same in the mixed form with as many sweeps as the exact arithmetic takes."""
    def run(**settings):
        sv = _indefinite(5, 4, gmres_restart=30, precision="mixed", **settings)
        x = _known(sv, "pressure_J")
        got, st = sv.gmres("pressure_J", np.zeros_like(x), sv.apply_operator("pressure_J", x))
        sv.close()
        return rel(got, x), st
    _, st = run(arith="exact")
    assert st["status"] == 0
    err, got = run(mixed_max_refine=st["refine_sweeps"])
    assert got["status"] == 0 and err <= 1e-7, (st, got, err)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_breakdown_leaves_newton_its_iterations(precision):
    """A Newton on negative enthalpies, whose Jacobian is not positive definite, with the iterations that
    the exact arithmetic takes (a linear problem: its solution lies above the floor)."""
    n = 6 * 5
    x = 1.0 + 0.1 * np.random.default_rng(5).standard_normal(n)
    cold = np.arange(0, n, 7)
    need = None
    for arith in ("exact", "fast"):
        more = {} if need is None else dict(Pnewton_max=need)
        sv = _newton_solver(6, 5, 2.0, arith=arith, precision=precision, gmres_restart=30, p_floor=1e-3, **more)
        q = sv.cons()
        q[4].reshape(-1)[cold] -= 40.0
        sv.set_buffer("Qe", q)
        sv.prepare_operator("pressure_L", 2.0 * 10.0 / 6)
        p, st = sv.nested_newton(np.full(n, 0.9), sv.apply_operator("pressure_L", x))
        assert st["status"] == 0 and rel(p, x) <= 1e-7, (arith, st, rel(p, x))
        need = st["newton_iters"] + 1  # the last iteration finds the residual small
        sv.close()


@pytest.mark.parametrize("kind", ["vortex", "blast"])
@pytest.mark.parametrize("op,settings", [("pressure_L", B_FORM), ("energy", ENERGY)])
@pytest.mark.parametrize("h", [4.0, 16.0])
def test_march_long_solves_are_as_accurate_as_gmres(op, settings, kind, h):
    """Solves of a hundred steps and more (condition numbers of 1e3 to 1e5): conjugate gradients stop on their
    recurrence residual however many they take, restarted GMRES (the exact arithmetic) forms b - A x at every
    restart.  The error is no larger than GMRES's, whose residual meets the same tolerance."""
    err = []
    for arith in ("exact", "fast"):
        sv, prob = _solver(kind, 64, 63, dict(settings, arith=arith))
        sv.prepare_operator(op, h * min(prob.dx, prob.dy))
        x = 1.0 + 0.3 * _known(sv, op)
        got, st = sv.gmres(op, np.zeros_like(x), sv.apply_operator(op, x))
        assert st["status"] == 0 and st["gmres_iters"] > 100, st
        err.append(rel(got, x))
        sv.close()
    assert err[1] <= err[0], err


@pytest.mark.parametrize("op,settings", [("pressure_L", B_FORM), ("energy", ENERGY)])
@pytest.mark.parametrize("kind,nx,ny,restart", [("vortex", 6, 5, 30), ("blast", 5, 6, 30), ("blast", 63, 41, 2)])
def test_a_cap_that_gmres_stays_below_is_no_refusal(op, settings, kind, nx, ny, restart):
    """Conjugate gradients can need a few steps more than GMRES, which minimises the residual's norm: a solve
    with as many restarts as the exact arithmetic takes still ends.  Thirty unknowns are one cycle of thirty.
    Tolerance: the stopping tolerance 1e-13 times the condition number, below 1e5."""
    need, steps = None, 30.0 if nx < 30 else 1.0
    for arith in ("exact", "fast"):
        more = {} if need is None else dict(gmres_max_restarts=need)
        sv, prob = _solver(kind, nx, ny, dict(settings, arith=arith, gmres_restart=restart, **more))
        sv.prepare_operator(op, steps * min(prob.dx, prob.dy))
        x = _known(sv, op)
        got, st = sv.gmres(op, np.zeros_like(x), sv.apply_operator(op, x))
        assert st["status"] == 0 and rel(got, x) <= 1e-8, (arith, need, st, rel(got, x))
        need = st["gmres_restarts"]
        sv.close()


@pytest.mark.parametrize("steps", [10.0, 30.0, 100.0])
def test_a_cap_that_newtons_gmres_stays_below_is_no_refusal(steps):
    """The same for the Jacobian solves of the nested Newton (a linear problem, solution above the floor)."""
    for arith in ("exact", "fast"):
        sv, prob = _solver("blast", 5, 6, dict(B_FORM, arith=arith, gmres_restart=30, gmres_max_restarts=1, p_floor=1e-6))
        sv.prepare_operator("pressure_L", steps * min(prob.dx, prob.dy))
        x = 1.0 + 0.1 * _known(sv, "pressure_L")
        p, st = sv.nested_newton(np.full(sv.N, 0.9), sv.apply_operator("pressure_L", x))
        assert st["status"] == 0 and rel(p, x) <= 1e-6, (arith, st, rel(p, x))
        sv.close()


@pytest.mark.parametrize("kind", ["vortex", "blast"])
@pytest.mark.parametrize("op,settings", [("pressure_L", B_FORM), ("energy", ENERGY)])
@pytest.mark.parametrize("restart", [2, 5, 12, 25])
def test_march_mixed_form_refines_ill_conditioned_systems(op, settings, kind, restart):
    """The mixed form within its fifty sweeps, however few residuals the inner solves keep.  Tolerance:
    mixed_outer_tol = 1e-10 times a condition number below 1e4."""
    for steps in (3.0, 10.0):
        sv, prob = _solver(kind, 143, 109, dict(settings, precision="mixed", mixed_solves=7, gmres_restart=restart))
        sv.prepare_operator(op, steps * min(prob.dx, prob.dy))
        x = _known(sv, op)
        got, st = sv.gmres(op, np.zeros_like(x), sv.apply_operator(op, x))
        assert st["status"] == 0 and rel(got, x) <= 1e-6, (steps, st, rel(got, x))
        sv.close()


def test_mixed_newton_keeps_pressures_above_a_small_floor():
    """A floor of 1e-8 beside a Newton tolerance of 1e-8 on 64 random fields: the mixed form leaves no converged
    solve with a pressure below theta p_floor where FP64 leaves none (IMEX_POSITIVITY), and takes at least as many
    of the fields' steps as the mixed GMRES does (the exact arithmetic).  An FP32 update is off by about the floor
    where it brings a pressure up from far below, so on either form some active sets flip until Pnewton_max."""
    base = dict(recon="ENO3", magfield="UnStaggerCT", add_pvisc="AlfvenSpeedp", add_bvisc=0, floor_on=1, p_floor=1e-8,
                theta=0.5, GMREStol=1e-13, y_bc="y_Transmissive", mixed_solves=5)
    forms = (dict(precision="fp64"), dict(precision="mixed", arith="exact"), dict(precision="mixed"))
    status = []
    for n in range(24, 72, 3):
        for seed in (1, 2, 3, 4):
            prob = random_field(n, seed=seed)
            prob.settings = {}
            status.append([])
            for more in forms:
                sv = ix.Solver.for_problem(prob, 3, dict(base, **more))
                try:
                    for _ in range(2):
                        sv.step()
                    status[-1].append(0)
                except ix.ImexError as e:
                    status[-1].append(e.status)
                sv.close()
    assert not [s for s in status if s[0] == 0 and s[2] == 7], status
    done = [sum(s[k] == 0 for s in status) for k in range(3)]
    assert done[0] >= 50 and done[2] >= done[1], done


@pytest.mark.parametrize("nx,ny,restart", [(393, 255, 25), (4100, 25, 25), (25, 4100, 25), (393, 255, 1), (393, 255, 3),
                                           (393, 255, 30)])
def test_march_a_form_of_large_contexts(nx, ny, restart):
    """The FP64 A form from the 100 thousand cells where one context's solve marches: a strip's width and one column
    past it, few long and many short runs, Krylov spaces below and past the ring."""
    sv, prob = _solver("sheet", nx, ny, dict(A_FORM, gmres_restart=restart))
    sv.prepare_operator("magnetic_A", 2.0 * min(prob.dx, prob.dy))
    x = _known(sv, "magnetic_A")
    got, st = sv.gmres("magnetic_A", np.zeros_like(x), sv.apply_operator("magnetic_A", x))
    assert st["status"] == 0 and rel(got, x) <= 1e-10, (st, rel(got, x))
    sv.close()
