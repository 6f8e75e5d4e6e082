"""BiCGSTAB's recurrence on upwind momentum matrices without relaxation: the residual vanishes on the
support of the first one, where r0.r is right only if it is taken from the updated residual. The
textbook recurrence takes 1,900 to 4,500 iterations on these systems (160 perturbed right-hand
sides; in the one-launch solve, which scales by D^-1 as it goes, single ones up to 10,800); with r0.r
as a difference of dots most of them do not converge within the default cap of 2 n = 20,000."""
import ctypes

import numpy as np
import pytest

from prism_b200 import _abi as A
from prism_b200 import api
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def systems():
    """Both momentum systems of the fourth SIMPLE step of a 100^2 cavity, urf 1."""
    import prism_b200
    lib = prism_b200.lib()
    mesh, U, p, nu, mdot, eqs = cases.cavity(100, lib)
    driver = api.IncompressibleSIMPLE(api.SIMPLEControls(momentum_urf=1.0), solver=api.BiCGSTAB())
    for _ in range(3):
        driver.step(eqs, U, mdot, p)
    ex, out = mesh.export(), []
    for c in (0, 1):
        eqs[c].zero_out_coeffs()
        eqs[c].update_coeffs()
        values, rhs = eqs[c].system()
        out.append((ex["csr_rowptr"].astype(np.int64), ex["csr_col"].astype(np.int64), values, rhs, U.values()[c]))
    return out


# caps beyond 2^20 run the ordinary iteration, kernel by kernel, others the one-launch solve
@pytest.mark.parametrize("cap", [0, (1 << 20) + 1])
@pytest.mark.parametrize("component", [0, 1])
def test_converges_like_the_textbook_recurrence(gpu, systems, component, cap):
    rowptr, col, values, rhs, guess = systems[component]
    o = api.BiCGSTAB(krylov_tol=1e-12, preconditioner="jacobi", krylov_max_iter=cap).opts(gpu)
    for seed in range(4):
        b = rhs * (1 + 1e-13 * np.random.default_rng(seed).normal(size=len(rhs)))
        x, r = guess.copy(), A.SolveResult()
        gpu.check(gpu.solve_csr(len(b), rowptr.ctypes.data_as(A.pi64), col.ctypes.data_as(A.pi64), api._f64p(values),
                                api._f64p(b), api._f64p(x), ctypes.byref(o), ctypes.byref(r)))
        print(f"component {component}, cap {cap}: {r.krylov_iterations} iterations, status {r.status}")
        assert r.status == A.OK and r.krylov_iterations <= 2 * len(b)
