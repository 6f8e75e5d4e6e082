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
        assert all(a.krylov_iterations < r.krylov_iterations for r, a in zip(res, again))
