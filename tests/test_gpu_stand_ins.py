"""Solves by smoothed aggregation that stand in for the method that was asked for: what they
leave as it was (the caller's choices and caps, the next solve) when one of them fails."""
import ctypes

import numpy as np
import pytest

from prism_b200 import _abi as A
from prism_b200 import api, meshgen
from tests import cases
from tests.test_gpu_smoothed import diffusion

pytestmark = pytest.mark.gpu


def counted(lib, f):
    """f() and the kernels it launched."""
    prof = A.Profile()
    lib.check(lib.profile_start(0))
    r = f()
    lib.check(lib.profile_stop(ctypes.byref(prof)))
    return r, prof.kernel_launches


def solve(solver, eqn, T, n_iter=1, eps=0.0):
    T.set_values(np.zeros(len(T.values())))
    return solver.solve(eqn, n_iter, eps)


def indefinite(n):
    """A few negative diffusivities: smoothed aggregation diverges, Jacobi-BiCGSTAB converges."""
    k = np.ones(n)
    k[::97] = -0.2
    return k


@pytest.mark.parametrize("graph", [False, True])
def test_asked_for_multigrid_is_used(gpu, graph):
    """12,144 rows, the automatic solve gave up multigrid: AMG and flexible CG that are asked
    for by name still run (a V-cycle solve launches hundreds of kernels or a loop of them, the
    one-launch solve a handful) and take the iterations that they take on a fresh equation."""
    want = {}
    for given_up in (False, True):
        mesh, T, eqn, (kappa, f) = diffusion(meshgen.box_hex(24, 22, 23), gpu)
        good = kappa.values()
        if given_up:
            kappa.set_values(indefinite(mesh.n_cells))
            assert solve(api.BiCGSTAB(), eqn, T).status == A.OK
            kappa.set_values(good)
        for solver in (api.FCG(graph=graph), api.BiCGSTAB(preconditioner="amg", graph=graph)):
            for _ in range(2):  # the second as a graph
                r, kernels = counted(gpu, lambda: solve(solver, eqn, T))
                assert r.status == A.OK and kernels > 20 and r.krylov_iterations < 60
            if given_up and isinstance(solver, api.FCG):
                assert cases.rel_l2(T.values(), want) < 1e-8
            want = T.values() if not given_up else want


def test_flexible_cg_after_dominance_chose_jacobi(gpu):
    """39,304 rows whose automatic choice was Jacobi (a small time step), then a failed AMG
    solve: flexible CG solves the equation as it did before."""
    mesh = api.Mesh(meshgen.box_hex(34, 34, 34), cases.box_case({"T": {p: ("fixed", 0.0) for p in meshgen.PATCHES}}),
                    lib=gpu)
    T = api.Scalar("T", mesh, 0.0)
    T.set_history_size(1)
    T.update(np.zeros(mesh.n_cells))
    kappa = api.Scalar("kappa", mesh, 1.0)
    f = api.Scalar("f", mesh, np.random.default_rng(1).normal(size=mesh.n_cells))
    time = api.temporal.BackwardEuler(T, 1e-6)
    eqn = api.Transport(time, api.diffusion.NonCorrected(kappa, T), api.source.ConstantScalar(f))
    assert solve(api.BiCGSTAB(), eqn, T).status == A.OK
    eqn.set_time_step(1e3)
    kappa.set_values(indefinite(mesh.n_cells))
    solve(api.BiCGSTAB(preconditioner="amg", krylov_max_iter=1000), eqn, T)
    kappa.set_values(np.ones(mesh.n_cells))
    assert solve(api.FCG(), eqn, T).status == A.OK


@pytest.mark.parametrize("cap", [3, 40, 600, 1000])
@pytest.mark.parametrize("preconditioner", ["auto", "amg"])
def test_iteration_cap_is_kept(gpu, cap, preconditioner):
    """The stand-in's iterations count against the caller's cap, which bounds them together."""
    mesh, T, eqn, (kappa, f) = diffusion(meshgen.box_hex(24, 22, 23), gpu)
    kappa.set_values(indefinite(mesh.n_cells))
    r = solve(api.BiCGSTAB(preconditioner=preconditioner, krylov_max_iter=cap), eqn, T)
    assert r.krylov_iterations <= cap
    assert r.status == A.OK or cap < 600 or preconditioner == "amg"  # plain AMG diverges on it too


def heat(lib, shape, kappa, dt, seed=1):
    """Implicit heat conduction on a box, one history step of zeros, walls held at 0."""
    mesh = api.Mesh(meshgen.box_hex(*shape), cases.box_case({"T": {p: ("fixed", 0.0) for p in meshgen.PATCHES}}),
                    lib=lib)
    T = api.Scalar("T", mesh, 0.0)
    T.set_history_size(1)
    T.update(np.zeros(mesh.n_cells))
    k = api.Scalar("kappa", mesh, kappa)
    f = api.Scalar("f", mesh, np.random.default_rng(seed).normal(size=mesh.n_cells))
    eqn = api.Transport(api.temporal.BackwardEuler(T, dt), api.diffusion.NonCorrected(k, T),
                        api.source.ConstantScalar(f))
    return mesh, T, eqn, (k, f)


@pytest.mark.parametrize("graph", [False, True])
def test_cap_of_every_step(gpu, graph):
    """The cap is each step's own: stand-ins that fail in one step after another (here because
    the first matrix, without couplings, left nothing to coarsen) are mended although their
    iterations add up to the cap."""
    mesh, T, eqn, (k, f) = heat(gpu, (700, 500, 1), 0.0, 1e-6)
    solver = api.BiCGSTAB(preconditioner="amg", krylov_max_iter=1000, graph=graph)
    assert solve(solver, eqn, T).status == A.OK
    k.set_values(np.random.default_rng(2).lognormal(0.0, 1.0, mesh.n_cells))
    eqn.set_time_step(1e6)
    r = solve(solver, eqn, T, 2)
    assert r.status == A.OK and r.iteration == 2 and r.krylov_rel_residual <= 1e-11
    assert r.krylov_iterations <= 2000


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("shape", [(24, 22, 23), (34, 33, 34)])
@pytest.mark.parametrize("where", ["source", "kappa", "guess"])
@pytest.mark.parametrize("first", [False, True])
def test_nan_in_one_call_does_not_change_the_next(gpu, shape, where, first, graph):
    """A call with a NaN ends as NONFINITE; the calls after it are, bit for bit, those of an
    equation that never saw one."""
    out = []
    for poisoned in (False, True):
        mesh, T, eqn, (kappa, f) = diffusion(meshgen.box_hex(*shape), gpu)
        solver = api.BiCGSTAB(graph=graph)
        for call in range(4):
            T.set_values(np.zeros(mesh.n_cells))
            field = {"source": f, "kappa": kappa, "guess": T}[where]
            good = field.values()
            if call == (0 if first else 2):
                if not poisoned:
                    continue
                bad = good.copy()
                bad[37] = np.nan
                field.set_values(bad)
            r = solver.solve(eqn, 3, 0.0)
            field.set_values(good) if where != "guess" else None
            assert r.status == (A.NONFINITE if call == (0 if first else 2) else A.OK)
        out.append((T.values(), r.krylov_iterations))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


def band(n, k, c):
    """Unit diagonal and k neighbours of weight c on either side: positive definite for the k and c
    used here (symbol >= 0.05), but D^-1 A reaches 1 + 2 k c, beyond what damped Jacobi smooths."""
    i = np.repeat(np.arange(n), 2 * k + 1)
    j = i + np.tile(np.arange(-k, k + 1), n)
    keep = (j >= 0) & (j < n)
    i, j = i[keep], j[keep]
    rowptr = np.zeros(n + 1, np.int64)
    np.add.at(rowptr, i + 1, 1)
    return np.cumsum(rowptr), j.astype(np.int64), np.where(i == j, 1.0, c), i


def solve_csr(lib, solver, rowptr, col, val, b):
    o, r, x = solver.opts(lib), A.SolveResult(), np.zeros(len(b))
    lib.check(lib.solve_csr(len(b), rowptr.ctypes.data_as(A.pi64), col.ctypes.data_as(A.pi64), api._f64p(val),
                            api._f64p(b), api._f64p(x), ctypes.byref(o), ctypes.byref(r)))
    return x, r


# condition numbers below 80: ||x - x*|| <= 80 ||r|| / ||A|| with ||r|| <= 1e-11 ||b|| (ten times the
# tolerance is accepted) is below 1e-8 ||x*||
@pytest.mark.parametrize("n, k, c", [(3000, 3, 0.2), (40000, 3, 0.3), (40000, 5, 0.2), (40000, 12, 0.1), (40000, 8, 0.2)])
def test_flexible_cg_beyond_dominance(gpu, n, k, c):
    rowptr, col, val, row = band(n, k, c)
    x = np.random.default_rng(0).normal(size=n)
    b = np.zeros(n)
    np.add.at(b, row, val * x[col])
    y, r = solve_csr(gpu, api.FCG(krylov_tol=1e-12), rowptr, col, val, b)
    assert r.status == A.OK and cases.rel_l2(y, x) < 1e-8
    assert r.krylov_iterations < 700 or c == 0.2 and k == 8


@pytest.mark.parametrize("graph", [False, True])
def test_flexible_cg_goes_back_to_amgs_own_cycle(gpu, graph):
    """A first matrix without couplings leaves smoothed aggregation nothing to coarsen; the next
    one's solve fails with it, and goes on with the plain cycle from the same guess."""
    mesh, T, eqn, (k, f) = heat(gpu, (700, 500, 1), 0.0, 1e-6)
    solver = api.FCG(graph=graph)
    assert solve(solver, eqn, T).status == A.OK
    k.set_values(np.random.default_rng(2).lognormal(0.0, 1.0, mesh.n_cells))
    eqn.set_time_step(1e6)
    for call in range(2):
        r = solve(solver, eqn, T)
        assert r.status == A.OK and r.krylov_rel_residual <= 1e-11
        assert r.krylov_iterations < (900 if call == 0 else 400)


def test_flexible_cg_beyond_dominance_takes_amgs_own_cycle(gpu):
    """No attempt with smoothed aggregation first, whose smoother does not reach that spectrum."""
    for n, k, c in ((3000, 3, 0.3), (40000, 5, 0.2)):
        rowptr, col, val, row = band(n, k, c)
        b = np.random.default_rng(0).normal(size=n)
        x, r = solve_csr(gpu, api.FCG(krylov_tol=1e-12), rowptr, col, val, b)
        assert r.status == A.OK and r.krylov_iterations < 100


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("preconditioner", ["auto", "amg"])
@pytest.mark.parametrize("first", [False, True])
def test_dominance_is_looked_at_again(gpu, preconditioner, graph, first):
    """An equation with negative diffusivities for two solves (its first, or later ones) gets its
    smoothed-aggregation solve back once they are gone, bit for bit that of an equation that never
    had them."""
    out = []
    for had in (False, True):
        mesh, T, eqn, (kappa, f) = diffusion(meshgen.box_hex(24, 22, 23), gpu)
        solver = api.BiCGSTAB(preconditioner=preconditioner, graph=graph)
        good = kappa.values()
        if not first:
            assert solve(solver, eqn, T).status == A.OK
        if had:
            kappa.set_values(indefinite(mesh.n_cells))
            for _ in range(2):
                r = solve(solver, eqn, T)
                assert r.status == A.OK or preconditioner == "amg"  # plain AMG diverges
            kappa.set_values(good)
        for _ in range(2):
            r = solve(solver, eqn, T)
            assert r.status == A.OK
        out.append((T.values(), r.krylov_iterations))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("solver", [api.BiCGSTAB, api.FCG])
def test_structure_of_another_matrix_is_built_anew(gpu, solver, graph):
    """Smoothed aggregation keeps the first matrix's aggregates. Where they are no use for a later
    matrix (the first had no couplings), the failed solve builds them anew; the solves after it
    are, bit for bit, those of an equation that began with the later matrix."""
    out = []
    for began in (False, True):
        mesh, T, eqn, (k, f) = heat(gpu, (700, 500, 1), 0.0, 1e-6)
        s = solver(preconditioner="amg", graph=graph)
        if began:
            assert solve(s, eqn, T).status == A.OK
        k.set_values(np.random.default_rng(2).lognormal(0.0, 1.0, mesh.n_cells))
        eqn.set_time_step(1e6)
        for call in range(3):
            r = solve(s, eqn, T)
            assert r.status == A.OK and (r.krylov_iterations < 60 or began and call == 0)
        out.append((T.values(), r.krylov_iterations))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


@pytest.mark.parametrize("clear", [True, False])
def test_fixed_point_with_coefficients_left_over(gpu, clear):
    """The first solve of a fixed point assembles onto what update_coeffs() left (here of a uniform
    coefficient, a million times larger), the next ones, with cleared coefficients, another matrix:
    their multigrid values are their own (sigma 2: a uniform coefficient's hierarchy would take
    some hundred iterations where its own takes a few tens). Without clearing, every solve has
    another matrix."""
    mesh, T, eqn, (kappa, f) = diffusion(meshgen.box_hex(34, 33, 32), gpu)
    kappa.set_values(np.full(mesh.n_cells, 1e6))
    eqn.update_coeffs()
    kappa.set_values(np.random.default_rng(5).lognormal(0.0, 2.0, mesh.n_cells))
    o = api.BiCGSTAB(preconditioner="amg").opts(gpu, n_iter=1, eps=0.0, clear_coeffs=clear)
    r = A.FixedPointResult()
    gpu.check(gpu.adjoint_forward(eqn.h, ctypes.byref(o), 3, 0.0, ctypes.byref(r)))
    print(f"{r.krylov_iterations} iterations in {r.outer_iterations} solves")
    assert r.status == A.OK and r.krylov_iterations < 120


def bicgstab_iterations(mesh, vals, b, tol):
    """Iterations of BiCGSTAB with the Jacobi preconditioner (van der Vorst 1992) on the exported system."""
    ex = mesh.export()
    rp, col = ex["csr_rowptr"], ex["csr_col"]
    row = np.repeat(np.arange(len(b)), np.diff(rp))
    diag = np.empty(len(b))
    diag[row[row == col]] = vals[row == col]
    mul = lambda v: np.bincount(row, vals * v[col], len(b))
    r = b.copy()
    r0, rho, p = r.copy(), r @ r, r.copy()
    for k in range(1, 2 * len(b)):
        v = mul(p / diag)
        alpha = rho / (r0 @ v)
        s = r - alpha * v
        t = mul(s / diag)
        w = (t @ s) / (t @ t)
        r = s - w * t
        if np.linalg.norm(r) <= tol * np.linalg.norm(b):
            return k
        rho, old = r0 @ r, rho
        p = r + (rho / old) * (alpha / w) * (p - w * v)
    return k


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("unv", [lambda: meshgen.box_tet(8, 8, 8), lambda: meshgen.box_tet(14, 14, 14), lambda: meshgen.box_hex(40, 40, 1)],
                         ids=["tet8", "tet14", "quad40"])
def test_cap_that_was_enough_for_bicgstab(gpu, unv, graph):
    """Conjugate gradients take its place in the one-launch solve: k of BiCGSTAB's iterations allow 2k of theirs,
    with the same number of products (6% over for rounding, which moves BiCGSTAB's count)."""
    mesh, T, eqn, keep = diffusion(unv(), gpu)
    eqn.update_coeffs()
    vals, b = eqn.system()
    eqn.zero_out_coeffs()
    k = bicgstab_iterations(mesh, np.asarray(vals), np.asarray(b).reshape(-1)[:mesh.n_cells], 1e-12)
    cap = int(1.06 * k) + 1
    r = solve(api.BiCGSTAB(preconditioner="jacobi", krylov_max_iter=cap, krylov_tol=1e-12, graph=graph), eqn, T)
    print(f"BiCGSTAB {k}, here {r.krylov_iterations}")
    assert r.status == A.OK and r.krylov_iterations <= cap


@pytest.mark.parametrize("graph", [False, True])
def test_cap_that_was_enough_with_amg(gpu, graph):
    """63,888 tetrahedra: 22 iterations of BiCGSTAB with amg's cycle, 26 of flexible CG (13 pairs)."""
    mesh, T, eqn, (kappa, f) = diffusion(meshgen.box_tet(22, 22, 22), gpu)
    kappa.set_values(np.ones(mesh.n_cells))
    solver = api.BiCGSTAB(preconditioner="amg", krylov_max_iter=24, graph=graph)
    for _ in range(3):
        r = solve(solver, eqn, T)
        assert r.status == A.OK and r.krylov_iterations <= 24
