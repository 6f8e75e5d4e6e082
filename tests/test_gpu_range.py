"""FP32 cycles inside FP64 solves: sources far below and above FP32's range (2^-140 is 7e-43, 2^140
is 1e42) are solved like those of ordinary size. Every operation of the FP64 recurrences scales
exactly by a power of two, and so does the cycle while its vectors stay within the range: the
solutions are the same bits."""
import numpy as np
import pytest

from prism_b200 import _abi as A
from prism_b200 import api, meshgen
from tests import cases
from tests.test_gpu_smoothed import diffusion

pytestmark = pytest.mark.gpu
POWERS = [-140, -100, -70, 90, 140]


@pytest.mark.parametrize("solver", [api.BiCGSTAB(), api.BiCGSTAB(preconditioner="amg"), api.FCG(), api.FCG(graph=True)],
                         ids=["auto", "amg", "fcg", "fcg_graph"])
@pytest.mark.parametrize("shape", [(24, 22, 23), (211, 190, 1)])
def test_symmetric(gpu, shape, solver):
    mesh, T, eqn, (kappa, f) = diffusion(meshgen.box_hex(*shape), gpu)
    source, want = f.values(), None
    for e in [0] + POWERS:
        f.set_values(source * 2.0 ** e)
        for _ in range(2):
            T.set_values(np.zeros(mesh.n_cells))
            r = solver.solve(eqn, 1, 0.0)
            assert r.status == A.OK
        want = (T.values(), r.krylov_iterations) if want is None else want
        assert np.array_equal(T.values() * 2.0 ** -e, want[0]) and r.krylov_iterations == want[1]


@pytest.mark.parametrize("graph", [False, True])
def test_convection(gpu, graph):
    want = None
    for e in [0] + POWERS:
        case = cases.box_case({"T": {"left": ("fixed", 2.0 ** e), "right": ("fixed", 0.0)}, "U": {}})
        mesh = api.Mesh(meshgen.box_hex(34, 33, 32, jitter=0.2, seed=2), case, lib=gpu)
        c = mesh.export()["cell_center"]
        U = api.Vector("U", mesh, np.stack([np.sin(np.pi * c[0]) * np.cos(np.pi * c[1]),
                                            -np.cos(np.pi * c[0]) * np.sin(np.pi * c[1]), np.zeros(mesh.n_cells)]))
        T, k = api.Scalar("T", mesh, 0.0), api.Scalar("kappa", mesh, 1e-2)
        eqn = api.Transport(api.convection.Upwind(U, T), api.diffusion.NonCorrected(k, T))
        for _ in range(2):
            T.set_values(np.zeros(mesh.n_cells))
            r = api.BiCGSTAB(preconditioner="amg", graph=graph).solve(eqn, 1, 0.0)
            assert r.status == A.OK
        want = (T.values(), r.krylov_iterations) if want is None else want
        assert np.array_equal(T.values() * 2.0 ** -e, want[0]) and r.krylov_iterations == want[1]


def test_batch(gpu):
    """Each system of its own size."""
    want = None
    for shift in range(len(POWERS) + 1):
        powers = np.roll([0] + POWERS, shift)[:4]
        probs = [cases.diffusion_box(N, gpu, seed=70 + i) for i, N in enumerate([20, 17, 11, 9])]
        for p, e in zip(probs, powers):
            p["f"].set_values(p["f"].values() * 2.0 ** e)
        res = api.BatchSolver(api.BiCGSTAB(precision=A.PREC_FP64), lib=gpu).solve([p["eqn"] for p in probs])
        assert all(r.status == A.OK for r in res)
        got = [(p["T"].values() * 2.0 ** -e, r.krylov_iterations) for p, e, r in zip(probs, powers, res)]
        want = got if want is None else want
        for (x, its), (y, its_y) in zip(got, want):
            assert np.array_equal(x, y) and its == its_y


SCRIPT = """
import sys
sys.path.insert(0, {root!r})
import numpy as np
import prism_b200
from prism_b200 import api, meshgen
from tests import cases
from tests.test_gpu_smoothed import diffusion
lib = prism_b200.lib()
mesh, T, eqn, keep = diffusion(meshgen.box_hex(34, 33, 32), lib)
a = api.BiCGSTAB().solve(eqn, 1, 0.0)
mesh2, T2, U, eqn2 = cases.transport_c3(32, lib, conv="Upwind")
b = api.BiCGSTAB(preconditioner="amg").solve(eqn2, 1, 0.0)
probs = [cases.diffusion_box(N, lib, seed=N) for N in (20, 21)]
c = api.BatchSolver(api.BiCGSTAB(precision=0), lib=lib).solve([p["eqn"] for p in probs])
its = [r.krylov_iterations for r in [a, b] + c]
np.savez({path!r}, its=its, T=T.values(), T2=T2.values(), b0=probs[0]["T"].values())
"""


def test_fp64_cycles_on_request(tmp_path):
    """PRISM_FCG_PREC=fp64 (read once per process): no FP32 cycle inside an FP64 solve. Users'
    equations then run as with PRISM_PRESSURE_SOLVER=bicgstab, by BiCGSTAB with amg's FP64 cycle,
    and batches by BiCGSTAB."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = {}
    for name, env in (("default", {}), ("fp64", {"PRISM_FCG_PREC": "fp64"}), ("plain", {"PRISM_PRESSURE_SOLVER": "bicgstab"})):
        path = str(tmp_path / (name + ".npz"))
        subprocess.run([sys.executable, "-c", SCRIPT.format(root=root, path=path)], env=dict(os.environ, **env),
                       check=True, timeout=300)
        out[name] = np.load(path)
    for field in ("T", "T2"):
        assert np.array_equal(out["fp64"][field], out["plain"][field])
    for field in ("T", "T2", "b0"):
        assert cases.rel_l2(out["fp64"][field], out["default"][field]) < 1e-8
    assert np.all(out["fp64"]["its"][2:] > 2 * out["default"]["its"][2:])
