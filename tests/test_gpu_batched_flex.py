"""Batches large enough for flexible CG over the block-diagonal matrix: what a call promises
(tolerance, iteration cap, independence of the systems from one another)."""
import numpy as np
import pytest

from prism_b200 import _abi as A
from prism_b200 import api
from tests import cases

pytestmark = pytest.mark.gpu


def batch(lib, sizes, **opts):
    probs = [cases.diffusion_box(N, lib, seed=70 + i) for i, N in enumerate(sizes)]
    return probs, api.BatchSolver(api.BiCGSTAB(**opts), lib=lib)


def solve(bs, probs):
    for p in probs:
        p["T"].set_values(np.zeros(p["mesh"].n_cells))
    return bs.solve([p["eqn"] for p in probs])


@pytest.mark.parametrize("precision", [A.PREC_MIXED, A.PREC_FP64])
@pytest.mark.parametrize("tol", [1e-12, 1e-14, 1e-15])
@pytest.mark.parametrize("sizes", [[20, 20], [24, 17, 31], [40, 33, 16, 9]])
def test_residuals_meet_the_tolerance(gpu, sizes, tol, precision):
    """OK means ||b - A x|| <= krylov_tol ||b||, down to a few units of the last place."""
    probs, bs = batch(gpu, sizes, precision=precision, krylov_tol=tol)
    for _ in range(2):
        res = solve(bs, probs)
        assert all(r.status == A.OK and r.krylov_rel_residual <= tol for r in res), res


def indefinite(p):
    """A few negative diffusivities: flexible CG fails on this system, BiCGSTAB solves it."""
    k = np.ones(p["mesh"].n_cells)
    k[::97] = -0.2
    p["kappa"].set_values(k)


@pytest.mark.parametrize("cap", [0, 40, 320, 600])
def test_iteration_cap_is_kept(gpu, cap):
    """Iterations of flexible CG are reported, and count against the caller's cap."""
    probs, bs = batch(gpu, [20, 21, 9], precision=A.PREC_FP64, krylov_max_iter=cap)
    indefinite(probs[1])
    res = solve(bs, probs)
    assert all(r.krylov_iterations <= cap for r in res) or cap == 0
    again = solve(bs, probs)  # without flexible CG
    if cap in (0, 600):
        assert all(r.status == A.OK for r in res + again)
    if cap == 0:
        assert again[1].krylov_iterations < res[1].krylov_iterations  # the system that failed


@pytest.mark.parametrize("where", ["source", "kappa", "guess"])
@pytest.mark.parametrize("when", [0, 1])
def test_nan_in_one_system(gpu, where, when):
    """A NaN ends its own system as NONFINITE. The others are solved, bit for bit as without it
    where their common multigrid hierarchy does not see it (kappa), and so are all in later calls."""
    out = []
    for poisoned in (False, True):
        probs, bs = batch(gpu, [20, 21, 9], precision=A.PREC_FP64)
        for call in range(3):
            for p in probs:
                p["T"].set_values(np.zeros(p["mesh"].n_cells))
            field = probs[1][{"source": "f", "kappa": "kappa", "guess": "T"}[where]]
            good = field.values()
            if call == when and poisoned:
                bad = good.copy()
                bad[5] = np.nan
                field.set_values(bad)
            res = bs.solve([p["eqn"] for p in probs])
            if call == when and poisoned and where != "guess":
                field.set_values(good)
            ok = [0, 2] if call == when and poisoned else [0, 1, 2]
            assert [i for i in range(3) if res[i].status == A.OK] == ok
            assert res[1].status == (A.OK if 1 in ok else A.NONFINITE)
            out.append(([p["T"].values() for p in probs], [r.krylov_iterations for r in res]))
    for call in range(3):
        (x, its), (y, its_y) = out[call], out[3 + call]
        for i in (0, 2) if call == when else (0, 1, 2):
            if call == when and where == "kappa":
                assert cases.rel_l2(y[i], x[i]) < 1e-8
            else:
                assert np.array_equal(x[i], y[i]) and its[i] == its_y[i]


def test_failed_system_does_not_change_later_calls(gpu):
    """Once its negative diffusivities are gone, a batch is again solved as one that never had them."""
    out = []
    for had in (False, True):
        probs, bs = batch(gpu, [20, 21, 9], precision=A.PREC_FP64)
        assert all(r.status == A.OK for r in solve(bs, probs))
        if had:
            good = probs[1]["kappa"].values()
            indefinite(probs[1])
            for _ in range(3):
                assert all(r.status == A.OK for r in solve(bs, probs))
            probs[1]["kappa"].set_values(good)
        for _ in range(2):
            res = solve(bs, probs)
            out.append(([p["T"].values() for p in probs], [r.krylov_iterations for r in res]))
    for x, its in out[1:]:
        assert its == out[0][1] and all(np.array_equal(a, b) for a, b in zip(x, out[0][0]))


def test_structure_of_other_matrices_is_built_anew(gpu):
    """Matrices without couplings in the first call left flexible CG nothing to coarsen: it fails
    in the second, and the third has a structure of its own."""
    from tests.test_gpu_stand_ins import heat
    probs = [heat(gpu, shape, 0.0, 1e-6) for shape in ((700, 500, 1), (20, 20, 20))]
    bs = api.BatchSolver(api.BiCGSTAB(precision=A.PREC_FP64), lib=gpu)
    for call in range(3):
        for mesh, T, eqn, (k, f) in probs:
            T.set_values(np.zeros(mesh.n_cells))
            if call == 1:
                k.set_values(np.random.default_rng(2).lognormal(0.0, 1.0, mesh.n_cells))
                eqn.set_time_step(1e6)
        res = bs.solve([p[2] for p in probs])
        assert all(r.status == A.OK and (call == 1 or r.krylov_iterations < 60) for r in res)


def test_more_systems_than_the_coarsest_solve_holds(gpu):
    """130 systems leave 130 rows without couplings on the coarsest level, more than the dense
    inverse takes: damped Jacobi sweeps solve it, and the fused tail is off."""
    sizes = [3 + i % 4 for i in range(126)] + [9, 1, 2, 11]
    probs, bs = batch(gpu, sizes, precision=A.PREC_FP64, krylov_tol=1e-13)
    assert sum(N ** 3 for N in sizes) >= 8192
    res = solve(bs, probs)
    assert all(r.status == A.OK and r.krylov_rel_residual <= 1e-13 and r.krylov_iterations < 40 for r in res)
    for i in (0, 1, 2, 3, 126, 127, 128, 129):
        q = cases.diffusion_box(sizes[i], gpu, seed=70 + i)
        api.BiCGSTAB(krylov_tol=1e-13, preconditioner="jacobi").solve(q["eqn"], 1, 0.0)
        assert cases.rel_l2(probs[i]["T"].values(), q["T"].values()) < 1e-8


def test_guess_is_back_where_the_cap_ends_a_failed_system(gpu):
    """A breakdown at the caller's cap leaves no iterations for BiCGSTAB: the field is the guess when
    the call's own residuals are taken from it, and when it returns."""
    probs, bs = batch(gpu, [20, 21, 9], precision=A.PREC_FP64, krylov_max_iter=5)
    indefinite(probs[1])
    for p in probs:
        p["T"].set_values(np.full(p["mesh"].n_cells, 0.25))
    res = bs.solve([p["eqn"] for p in probs])
    assert all(r.krylov_iterations <= 5 for r in res)
    if res[1].status == A.BREAKDOWN:
        assert np.all(probs[1]["T"].values() == 0.25)
        assert res[1].final_residual == res[1].initial_residual


def test_refused_equation_leaves_the_batch_usable(gpu):
    """An equation without a boundary handler ends the call while the others' residuals are on
    their way to the batch's pinned memory, which the next, larger call allocates anew."""
    from prism_b200 import PrismError
    from tests.test_failures import no_handler_case
    refused = no_handler_case(gpu)[-1]
    probs, bs = batch(gpu, [20, 21, 9], precision=A.PREC_FP64)
    for _ in range(3):
        with pytest.raises(PrismError) as e:
            bs.solve([probs[0]["eqn"], refused])
        assert e.value.status == A.NO_BC_HANDLER
    probs[0]["eqn"].zero_out_coeffs()  # it was assembled before the refusal
    got = solve(bs, probs), [p["T"].values() for p in probs]
    probs, bs = batch(gpu, [20, 21, 9], precision=A.PREC_FP64)
    want = solve(bs, probs), [p["T"].values() for p in probs]
    assert all(np.array_equal(a, b) for a, b in zip(got[1], want[1]))
    assert [r.initial_residual for r in got[0]] == [r.initial_residual for r in want[0]]
