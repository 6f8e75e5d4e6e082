"""Flexible CG with the smoothed-aggregation cycle, at the sizes where its levels, tail and
coarsest solve change: one dense level, levels inside the fused tail only, levels above it,
thin and ragged boxes, tetrahedra, strongly varying coefficients and rows without couplings."""
import numpy as np
import pytest

import oracle
import prism_b200
from prism_b200 import api, meshgen
from tests import cases

pytestmark = pytest.mark.gpu


def diffusion(unv, lib, seed=1):
    """Lognormal kappa, normal source, walls held at 0."""
    case = cases.box_case({"T": {p: ("fixed", 0.0) for p in meshgen.PATCHES}})
    mesh = api.Mesh(unv, case, lib=lib)
    rng = np.random.default_rng(seed)
    kappa = api.Scalar("kappa", mesh, rng.lognormal(0.0, 1.0, mesh.n_cells))
    f = api.Scalar("f", mesh, rng.normal(0.0, 1.0, mesh.n_cells))
    T = api.Scalar("T", mesh, 0.0)
    eqn = api.Transport(api.diffusion.NonCorrected(kappa, T), api.source.ConstantScalar(f))
    return mesh, T, eqn, (kappa, f)


# ||x - x*|| <= cond(A) ||r|| / ||A||: with ||r|| <= 1e-13 ||b|| and cond(A) below 1e5 at these
# sizes every pair of solutions agrees to 1e-8, the bound of the solved-field tests
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 2, 1), (96, 1, 1), (97, 1, 1), (10, 10, 1), (33, 31, 1), (90, 47, 1),
                                   (13, 11, 12)])
def test_matches_oracle(shape):
    out = []
    for lib, solver in ((prism_b200.lib(), api.FCG(krylov_tol=1e-13)), (oracle.lib(), api.BiCGSTAB())):
        mesh, T, eqn, keep = diffusion(meshgen.box_hex(*shape), lib)
        r = solver.solve(eqn, 1, 0.0)
        assert r.status == 0
        out.append(T.values())
    assert cases.rel_l2(out[0], out[1]) < 1e-8


@pytest.mark.parametrize("unv", [lambda: meshgen.box_hex(211, 190, 1), lambda: meshgen.box_hex(41, 38, 36),
                                 lambda: meshgen.box_tet(4, 5, 3), lambda: meshgen.box_tet(18, 17, 19)],
                         ids=["hex2d", "hex3d", "tet_small", "tet"])
def test_matches_bicgstab(unv):
    lib, out = prism_b200.lib(), []
    mesh, T, eqn, keep = diffusion(unv(), lib)
    for solver in (api.FCG(krylov_tol=1e-13), api.BiCGSTAB(krylov_tol=1e-13, preconditioner="jacobi"),
                   api.FCG(krylov_tol=1e-13)):
        T.set_values(np.zeros(mesh.n_cells))
        r = solver.solve(eqn, 1, 0.0)
        assert r.status == 0
        out.append(T.values())
    assert cases.rel_l2(out[0], out[1]) < 1e-8
    assert np.array_equal(out[0], out[2])  # the refreshed hierarchy is the built one


def test_rows_without_couplings():
    n = 200
    d = np.random.default_rng(2).uniform(1.0, 9.0, n)
    b = np.random.default_rng(3).normal(size=n)
    x = api.FCG(krylov_tol=1e-12).step(prism_b200.lib(), np.arange(n + 1), np.arange(n), d, np.zeros(n), b)
    assert np.allclose(x, b / d, rtol=1e-10, atol=0)
