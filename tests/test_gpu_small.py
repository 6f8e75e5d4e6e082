"""Whole solves in one launch (systems of up to 32,768 rows), at the edges of its blocks and
clusters: one row, part of a warp, one block of one and of two rows per thread, the first size
of each cluster shape, the last one, and one row past it (the ordinary path)."""
import numpy as np
import pytest

import prism_b200
from prism_b200 import _abi as A
from prism_b200 import api
from tests import cases

pytestmark = pytest.mark.gpu


def system(n, seed, wide, symmetric):
    """A diagonally dominant band matrix (half-bandwidth wide) with zero sums outside the ends."""
    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), 2 * wide + 1)
    j = i + np.tile(np.arange(-wide, wide + 1), n)
    keep = (j >= 0) & (j < n)
    i, j = i[keep], j[keep]
    v = -rng.uniform(0.5, 1.5, len(i))
    if symmetric:
        low, high = np.minimum(i, j), np.maximum(i, j)
        v = -(0.5 + ((low * 7919 + high * 104729) % 1009) / 1009.0)
    v[i == j] = 0.0
    diag = np.zeros(n)
    np.add.at(diag, i, -v)
    v[i == j] = diag[i[i == j]] * 1.1 + 0.1
    rowptr = np.zeros(n + 1, np.int64)
    np.add.at(rowptr, i + 1, 1)
    return np.cumsum(rowptr), j, v, i


# the oracle of a raw system is its own definition: b = A x* for a chosen x*, whose recovery
# to tol (1e-13) times the condition number (below 1e3: dominance 1.1) is held to 1e-9
@pytest.mark.parametrize("n", [1, 31, 256, 257, 1024, 1025, 4096, 4097, 16384, 16385, 32768, 32769])
@pytest.mark.parametrize("wide", [2, 5])
def test_recovers_the_solution(n, wide):
    rowptr, col, val, row = system(n, n + wide, wide, False)
    x = np.random.default_rng(n).normal(size=n)
    b = np.zeros(n)
    np.add.at(b, row, val * x[col])
    got = api.BiCGSTAB(krylov_tol=1e-13, preconditioner="jacobi").step(prism_b200.lib(), rowptr, col, val, np.zeros(n), b)
    assert cases.rel_l2(got, x) < 1e-9


@pytest.mark.parametrize("shape", [(5, 1, 1), (16, 16, 1), (32, 32, 1), (33, 31, 1), (21, 22, 23)])
def test_symmetric_equations_match_the_oracle(gpu, orc, shape):
    """Conjugate gradients on diffusion, with several outer steps and the record they return."""
    from prism_b200 import meshgen
    from tests.test_gpu_smoothed import diffusion
    out = {}
    for lib in (gpu, orc):
        mesh, T, eqn, keep = diffusion(meshgen.box_hex(*shape), lib)
        r = api.BiCGSTAB(krylov_tol=1e-13, preconditioner="jacobi" if lib is gpu else "auto").solve(eqn, 2, 1e-30)
        assert r.status == A.OK and r.iteration == 2
        out[lib] = T.values()
    assert cases.rel_l2(out[gpu], out[orc]) < 1e-8


def test_indefinite_symmetric_equation_falls_back(gpu, orc):
    """Negative diffusivities in a few cells: no M-matrix, so BiCGSTAB solves it, as in the reference."""
    from prism_b200 import meshgen
    from tests.test_gpu_smoothed import diffusion
    out = {}
    for lib in (gpu, orc):
        mesh, T, eqn, (kappa, f) = diffusion(meshgen.box_hex(9, 9, 9), lib)
        k = np.ones(mesh.n_cells)
        k[::50] = -0.1
        kappa.set_values(k)
        r = api.BiCGSTAB(krylov_tol=1e-13).solve(eqn, 1, 0.0)
        assert r.status == A.OK
        out[lib] = T.values()
    assert cases.rel_l2(out[gpu], out[orc]) < 1e-8


def test_zero_right_hand_side(gpu):
    n = 700
    rowptr, col, val, row = system(n, 3, 3, False)
    x = api.BiCGSTAB(preconditioner="jacobi").step(gpu, rowptr, col, val, np.ones(n), np.zeros(n))
    assert np.all(x == 0.0)


@pytest.mark.parametrize("shape", [(10, 10, 10), (15, 14, 13)])
@pytest.mark.parametrize("symmetric", [False, True])
def test_outer_steps_are_spread_over_launches(gpu, shape, symmetric):
    """One launch holds 2^20 iterations at most: with the largest cap a step each, with a third of
    it three, with a small one all; fields and records are the same, as a graph too."""
    import ctypes
    from prism_b200 import meshgen
    from tests.test_gpu_smoothed import diffusion
    runs = {}
    for cap in (0, (1 << 20) // 3, 1 << 20):
        for graph in (False, True):
            if symmetric:
                mesh, T, eqn, keep = diffusion(meshgen.box_hex(*shape), gpu)
            else:
                mesh, T, U, eqn = cases.transport_c3(shape[0], gpu, conv="Upwind")
            solver = api.BiCGSTAB(krylov_max_iter=cap, preconditioner="jacobi", graph=graph)
            solver.solve(eqn, 1, 0.0)
            T.set_values(np.zeros(mesh.n_cells))
            prof = A.Profile()
            gpu.check(gpu.profile_start(0))
            r = solver.solve(eqn, 7, 0.0)
            gpu.check(gpu.profile_stop(ctypes.byref(prof)))
            runs[cap, graph] = (T.values(), (r.status, r.iteration, r.krylov_iterations, r.initial_residual,
                                             r.final_residual, r.krylov_rel_residual), prof.kernel_launches)
    first = runs[0, False]
    assert first[1][:2] == (A.OK, 7)
    for x, record, launches in runs.values():
        assert np.array_equal(x, first[0]) and record == first[1]
    for graph in (False, True):
        assert [runs[cap, graph][2] - runs[0, graph][2] for cap in ((1 << 20) // 3, 1 << 20)] == [2, 6]
