"""Performance cases of the framework: what its users run, through the public API.

Each case is a whole call sequence of a user's program on one mesh: the fields go in from
pinned host memory, the solver calls run, and the resulting fields come back to pinned
host memory. Meshes, fields, equations and solver objects are made once by `prepare`, as
a program that solves again and again keeps them. Kinds:

  poisson    steady diffusion with a source and fixed wall values on a uniform box
  simple     SIMPLE outer iterations of the lid-driven cavity (2-D and 3-D)
  transport  steady convection-diffusion on a jittered hex box, one step of the solver
  transient  time steps of convection-diffusion on tetrahedra
  batch      many independent diffusion systems in one batched call
  adjoint    forward solve and discrete adjoint of steady diffusion on tetrahedra
"""
import numpy as np
import torch

import prism_b200
from prism_b200 import _abi as A
from prism_b200 import api, io, meshgen

WALLS = meshgen.PATCHES


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the steady Poisson problem of the reference's own test, at the size of the first
        # benchmark configuration: a small 2-D solve, bound by launches and latency
        {"name": "poisson_2d_128", "kind": "poisson", "nx": 128, "ny": 128, "nz": 1, "solver": "bicgstab"},
        # a 3-D potential / heat-conduction solve with the symmetric solver, odd and unequal edges
        {"name": "poisson_3d_97", "kind": "poisson", "nx": 97, "ny": 80, "nz": 89, "solver": "fcg"},
        # the smallest flow: the cavity as tutorials and tests run it, default solver options
        {"name": "simple_32", "kind": "simple", "nx": 32, "ny": 32, "nz": 1, "steps": 6, "graph": False},
        # a 3-D cavity (three momentum equations), ragged edges, default solver options
        {"name": "simple_3d_44", "kind": "simple", "nx": 44, "ny": 37, "nz": 41, "steps": 3, "graph": False},
        # the second benchmark configuration: 512 x 512 cavity, each outer iteration one graph
        {"name": "simple_512", "kind": "simple", "nx": 512, "ny": 512, "nz": 1, "steps": 3, "graph": True},
        # the headline workload of bench.py: the 2.1M-cell cavity
        {"name": "simple_1448", "kind": "simple", "nx": 1448, "ny": 1448, "nz": 1, "steps": 2, "graph": True},
        # scalar transport below the size where multigrid is chosen
        {"name": "transport_31", "kind": "transport", "nx": 31, "ny": 31, "nz": 31, "conv": "MUSCL",
         "grad": "green-gauss", "precision": "fp64"},
        # mixed precision (FP32 iterations, FP64 updates) on a mid-sized box, least-squares gradients
        {"name": "transport_71_mixed", "kind": "transport", "nx": 71, "ny": 64, "nz": 67, "conv": "LinearUpwind",
         "grad": "least-squares", "precision": "mixed"},
        # the third benchmark configuration: 128^3 skewed hexes, MUSCL, Green-Gauss
        {"name": "transport_128", "kind": "transport", "nx": 128, "ny": 128, "nz": 128, "conv": "MUSCL",
         "grad": "green-gauss", "precision": "fp64"},
        # time stepping on an unstructured mesh: assembly, gradients and a well-conditioned solve per step
        {"name": "transient_tet_17", "kind": "transient", "n": 17, "steps": 5},
        # a parameter study: independent systems of uneven sizes, mixed precision, one call
        {"name": "batch_24", "kind": "batch", "count": 24, "nmin": 16, "nmax": 48, "precision": "mixed"},
        # gradient of an objective with respect to conductivities and wall values
        {"name": "adjoint_tet_22", "kind": "adjoint", "n": 22},
    ]


def _loguniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    """One more case of the listed ranges (edges over their logarithm, odd ones among them)."""
    kind = rng.choice(["poisson", "poisson", "simple", "simple", "simple", "transport", "transport", "transient",
                       "batch", "adjoint"])
    if kind == "poisson":
        if rng.random() < 0.5:
            nx, ny, nz = _loguniform(rng, 24, 400), _loguniform(rng, 24, 400), 1
        else:
            nx, ny, nz = (_loguniform(rng, 12, 97) for _ in range(3))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "solver": rng.choice(["bicgstab", "bicgstab", "fcg"])}
    if kind == "simple":
        if rng.random() < 0.7:
            nx = _loguniform(rng, 24, 700)
            ny = max(16, int(nx * rng.uniform(0.7, 1.3)))
            nz = 1
        else:
            nx, ny, nz = (_loguniform(rng, 10, 56) for _ in range(3))
        cells = nx * ny * nz
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": 6 if cells < 8000 else 3,
                "graph": rng.random() < 0.5}
    if kind == "transport":
        nx, ny, nz = (_loguniform(rng, 14, 96) for _ in range(3))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "conv": rng.choice(["MUSCL", "LinearUpwind", "Upwind"]),
                "grad": rng.choice(["green-gauss", "least-squares"]), "precision": rng.choice(["fp64", "mixed"])}
    if kind == "transient":
        return {"kind": kind, "n": _loguniform(rng, 6, 32), "steps": rng.randint(2, 6)}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(4, 32), "nmin": rng.randint(8, 16), "nmax": rng.randint(20, 48),
                "precision": rng.choice(["mixed", "mixed", "fp64"])}
    return {"kind": kind, "n": _loguniform(rng, 8, 26)}


# ---------------------------------------------------------------- host buffers and case documents
def _pinned(a):
    """A pinned host copy of an array (the buffers a program moves fields through)."""
    a = np.ascontiguousarray(a, dtype=np.float64)
    t = torch.empty(a.size, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    out = t.numpy()
    out[:] = a.reshape(-1)
    return out


def _ptr(a):
    return a.ctypes.data_as(A.pf64)


def _box(bcs, info=None):
    fields = {f: {p: per.get(p, ("zero-gradient", None)) for p in WALLS} for f, per in bcs.items()}
    return io.Case.from_dict(WALLS, fields, info)


def _smooth(rng, x, y, z, amplitude=1.0, modes=4):
    """A smooth field: a few cosine modes of seeded amplitudes and phases."""
    out = np.zeros_like(x)
    for _ in range(modes):
        k = rng.integers(1, 4, 3)
        ph = rng.uniform(0.0, 2.0 * np.pi, 3)
        out += rng.normal() * np.cos(np.pi * k[0] * x + ph[0]) * np.cos(np.pi * k[1] * y + ph[1]) * \
            np.cos(np.pi * k[2] * z + ph[2])
    return amplitude * out


# ---------------------------------------------------------------- Poisson
def _poisson_inputs(case, seed):
    """Source per cell (smooth, with cell noise) and the wall values, one number per wall."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    z, y, x = np.meshgrid((np.arange(nz) + 0.5) / nz, (np.arange(ny) + 0.5) / ny, (np.arange(nx) + 0.5) / nx,
                          indexing="ij")
    f = _smooth(rng, x, y, z, 20.0) + rng.normal(0.0, 1.0, x.shape)
    return f.reshape(-1), {p: float(v) for p, v in zip(WALLS, rng.uniform(-1.0, 1.0, 6))}


def _lengths(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return (1.0, 1.0, 1.0 if nz > 1 else 1.0 / nx)


def _prepare_poisson(case, seed):
    lib = prism_b200.lib()
    f, walls = _poisson_inputs(case, seed)
    unv = meshgen.box_hex(case["nx"], case["ny"], case["nz"], _lengths(case))
    flat = case["nz"] == 1
    bcs = {p: ("symmetry", None) if flat and p in ("back", "front") else ("fixed", walls[p]) for p in WALLS}
    mesh = api.Mesh(unv, _box({"P": bcs}), lib=lib)
    P = api.Scalar("P", mesh, 0.0)
    S = api.Scalar("S", mesh, 0.0)
    kappa = api.Scalar("kappa", mesh, 1.0)
    eqn = api.Transport(api.diffusion.NonCorrected(kappa, P), api.source.ConstantScalar(S))
    solver = api.FCG(krylov_tol=1e-13) if case["solver"] == "fcg" else api.BiCGSTAB(krylov_tol=1e-13)
    return dict(case=case, lib=lib, mesh=mesh, P=P, S=S, kappa=kappa, eqn=eqn, solver=solver, f=_pinned(f),
                zero=_pinned(np.zeros(mesh.n_cells)), out=_pinned(np.zeros(mesh.n_cells)))


def _run_poisson(s):
    lib = s["lib"]
    s["S"].set_values(s["f"])
    s["P"].set_values(s["zero"])
    s["solver"].solve(s["eqn"], 1, 0.0)
    lib.check(lib.scalar_get_values(s["P"].h, _ptr(s["out"])))
    return s["out"]


def _exact_poisson(case, seed):
    """The seven-point system of the uniform box in 64 bits, solved in the eigenvectors of
    its one-dimensional parts."""
    f, walls = _poisson_inputs(case, seed)
    n = [case["nx"], case["ny"], case["nz"]]
    h = [l / m for l, m in zip(_lengths(case), n)]
    vol = h[0] * h[1] * h[2]
    b = f.reshape(n[2], n[1], n[0]) * vol
    parts = []
    for axis, (lo, hi) in enumerate((("left", "right"), ("bottom", "top"), ("back", "front"))):
        m, g = n[axis], vol / (h[axis] * h[axis])  # face area over distance
        T = np.zeros((m, m))
        i = np.arange(m - 1)
        T[i, i] += g
        T[i + 1, i + 1] += g
        T[i, i + 1] -= g
        T[i + 1, i] -= g
        if axis < 2 or n[2] > 1:
            T[0, 0] += 2.0 * g
            T[m - 1, m - 1] += 2.0 * g
            first, last = [slice(None)] * 3, [slice(None)] * 3
            first[2 - axis], last[2 - axis] = 0, m - 1
            b[tuple(first)] += 2.0 * g * walls[lo]
            b[tuple(last)] += 2.0 * g * walls[hi]
        parts.append(np.linalg.eigh(T))
    (lx, Qx), (ly, Qy), (lz, Qz) = parts
    t = np.einsum("kc,cba->kba", Qz.T, b)
    t = np.matmul(Qy.T[None], t)
    t = np.matmul(t, Qx)
    t /= lz[:, None, None] + ly[None, :, None] + lx[None, None, :]
    t = np.matmul(t, Qx.T)
    t = np.matmul(Qy[None], t)
    return np.einsum("kc,cba->kba", Qz, t).reshape(-1)


# ---------------------------------------------------------------- SIMPLE
def _prepare_simple(case, seed):
    lib = prism_b200.lib()
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    flat = nz == 1
    unv = meshgen.box_hex(nx, ny, nz, (1.0, 1.0, 1.0 / nx if flat else 1.0))
    wall = ("no-slip", [0.0, 0.0, 0.0])
    ub = {"top": ("fixed", [1.0, 0.0, 0.0]), "left": wall, "right": wall, "bottom": wall,
          "back": ("empty", None) if flat else wall, "front": ("empty", None) if flat else wall}
    pb = {"back": ("empty", None), "front": ("empty", None)} if flat else {}
    mesh = api.Mesh(unv, _box({"U": ub, "P": pb}), lib=lib)
    z, y, x = np.meshgrid((np.arange(nz) + 0.5) / nz, (np.arange(ny) + 0.5) / ny, (np.arange(nx) + 0.5) / nx,
                          indexing="ij")
    x, y, z = x.reshape(-1), y.reshape(-1), z.reshape(-1)
    # an earlier state of the flow: a vortex filling the cavity, disturbed by seeded modes
    sx, sy = np.sin(np.pi * x), np.sin(np.pi * y)
    a = rng.uniform(0.05, 0.2)
    U0 = np.stack([a * sx * sx * np.sin(2 * np.pi * y), -a * sy * sy * np.sin(2 * np.pi * x), np.zeros_like(x)])
    U0[0] += 0.02 * sx * sy * _smooth(rng, x, y, z)
    U0[1] += 0.02 * sx * sy * _smooth(rng, x, y, z)
    if not flat:
        U0[2] += 0.02 * sx * sy * np.sin(np.pi * z) * _smooth(rng, x, y, z)
    p0 = _smooth(rng, x, y, z, 0.01)
    U = api.Vector("U", mesh, U0)
    p = api.Scalar("P", mesh, p0)
    nu = api.Scalar("nu", mesh, 0.01 * rng.uniform(0.8, 1.25))
    mdot = U.clone()
    flux = _pinned(U.face_flux())
    eqs = [api.Transport(api.convection.Upwind(mdot, c), api.diffusion.Corrected(nu, c),
                         api.source.Gradient(p, k, A.SIGN_NEGATIVE))
           for k, c in enumerate([U.x(), U.y()] + ([] if flat else [U.z()]))]
    simple = api.IncompressibleSIMPLE(api.SIMPLEControls(),
                                      solver=api.BiCGSTAB(graph=case["graph"]))
    return dict(case=case, lib=lib, mesh=mesh, U=U, p=p, nu=nu, mdot=mdot, eqs=eqs, simple=simple, flux=flux,
                U0=_pinned(U0), p0=_pinned(p0), outU=_pinned(U0), outp=_pinned(p0))


def _run_simple(s):
    lib = s["lib"]
    s["U"].set_values(s["U0"])
    s["p"].set_values(s["p0"])
    s["mdot"].set_face_flux(s["flux"])
    for _ in range(s["case"]["steps"]):
        s["simple"].step(s["eqs"], s["U"], s["mdot"], s["p"])
    lib.check(lib.vector_get_values(s["U"].h, _ptr(s["outU"])))
    lib.check(lib.scalar_get_values(s["p"].h, _ptr(s["outp"])))
    return {"U": s["outU"], "p": s["outp"]}


# ---------------------------------------------------------------- scalar transport
def _prepare_transport(case, seed):
    lib = prism_b200.lib()
    rng = np.random.default_rng(seed)
    unv = meshgen.box_hex(case["nx"], case["ny"], case["nz"], jitter=0.2, seed=seed)
    doc = _box({"T": {"left": ("fixed", 1.0), "right": ("fixed", 0.0)}, "U": {}},
               {"T": {"gradScheme": "greenGauss"} if case["grad"] == "green-gauss" else {}, "U": {}})
    mesh = api.Mesh(unv, doc, lib=lib)
    c = mesh.export()["cell_center"]
    a = rng.uniform(0.8, 1.2)
    U = api.Vector("U", mesh, np.stack([a * np.sin(np.pi * c[0]) * np.cos(np.pi * c[1]),
                                        -a * np.cos(np.pi * c[0]) * np.sin(np.pi * c[1]), np.zeros(mesh.n_cells)]))
    T = api.Scalar("T", mesh, 0.0)
    kappa = api.Scalar("kappa", mesh, 1e-3)
    eqn = api.Transport(getattr(api.convection, case["conv"])(U, T), api.diffusion.Corrected(kappa, T))
    solver = api.BiCGSTAB(precision=A.PREC_MIXED if case["precision"] == "mixed" else A.PREC_FP64)
    scheme = A.GRAD_GREEN_GAUSS if case["grad"] == "green-gauss" else A.GRAD_LEAST_SQUARES
    return dict(case=case, lib=lib, mesh=mesh, U=U, T=T, kappa=kappa, eqn=eqn, solver=solver, scheme=scheme,
                zero=_pinned(np.zeros(mesh.n_cells)), out=_pinned(np.zeros(mesh.n_cells)))


def _run_transport(s):
    lib = s["lib"]
    s["T"].set_values(s["zero"])
    if s["scheme"] == A.GRAD_GREEN_GAUSS:
        s["T"].set_grad_scheme(s["scheme"])  # Green-Gauss sweeps start from the last gradients: begin from none
    s["solver"].solve(s["eqn"], 1, 0.0)
    lib.check(lib.scalar_get_values(s["T"].h, _ptr(s["out"])))
    return s["out"]


# ---------------------------------------------------------------- transient on tetrahedra
def _prepare_transient(case, seed):
    lib = prism_b200.lib()
    rng = np.random.default_rng(seed)
    unv = meshgen.box_tet(case["n"], case["n"], case["n"])
    mesh = api.Mesh(unv, _box({"T": {"left": ("fixed", 1.0), "right": ("fixed", 0.0)}, "U": {}}), lib=lib)
    c = mesh.export()["cell_center"]
    U = api.Vector("U", mesh, np.stack([np.sin(np.pi * c[0]) * np.cos(np.pi * c[1]),
                                        -np.cos(np.pi * c[0]) * np.sin(np.pi * c[1]), np.zeros(mesh.n_cells)]))
    T0 = 0.5 + _smooth(rng, c[0], c[1], c[2], 0.2)
    T = api.Scalar("T", mesh, T0)
    T.set_history_size(1)
    kappa = api.Scalar("kappa", mesh, 1e-2 * rng.uniform(0.5, 2.0))
    eqn = api.Transport(api.temporal.BackwardEuler(T, 0.5 / case["n"]), api.convection.Upwind(U, T),
                        api.diffusion.Corrected(kappa, T))
    return dict(case=case, lib=lib, mesh=mesh, U=U, T=T, kappa=kappa, eqn=eqn, solver=api.BiCGSTAB(),
                T0=_pinned(T0), out=_pinned(T0))


def _run_transient(s):
    lib, T = s["lib"], s["T"]
    T.set_values(s["T0"])
    T.update_prev_time_steps()
    for _ in range(s["case"]["steps"]):
        s["solver"].solve(s["eqn"], 2, 1e-20)  # two deferred-correction passes per time step
        T.update_prev_time_steps()
    lib.check(lib.scalar_get_values(T.h, _ptr(s["out"])))
    return s["out"]


# ---------------------------------------------------------------- batched systems
def _batch_sizes(case):
    """Edge lengths of the systems: the mix of sizes is the case's, the coefficients are the seed's."""
    rng = np.random.default_rng(4)
    lo, hi = np.log(case["nmin"]), np.log(case["nmax"])
    return [int(round(float(np.exp(rng.uniform(lo, hi))))) for _ in range(case["count"])]


def _batch_coefficients(case, seed):
    """(N, conductivity per cell, source per cell) of every system."""
    rng = np.random.default_rng(seed)
    for N in _batch_sizes(case):
        kappa = rng.lognormal(0.0, 1.0, N ** 3)
        yield N, kappa, rng.normal(0.0, 1.0, N ** 3)


def _prepare_batch(case, seed):
    lib = prism_b200.lib()
    doc = _box({"T": {p: ("fixed", 0.0) for p in WALLS}})
    probs = []
    for N, kappa0, f0 in _batch_coefficients(case, seed):
        mesh = api.Mesh(meshgen.box_hex(N, N, N), doc, lib=lib)
        kappa = api.Scalar("kappa", mesh, kappa0)
        f = api.Scalar("f", mesh, f0)
        T = api.Scalar("T", mesh, 0.0)
        eqn = api.Transport(api.diffusion.Corrected(kappa, T), api.source.ConstantScalar(f))
        probs.append(dict(mesh=mesh, kappa=kappa, f=f, T=T, eqn=eqn, zero=_pinned(np.zeros(mesh.n_cells)),
                          out=_pinned(np.zeros(mesh.n_cells))))
    precision = A.PREC_MIXED if case["precision"] == "mixed" else A.PREC_FP64
    solver = api.BatchSolver(api.BiCGSTAB(precision=precision, krylov_tol=1e-12), lib=lib)
    return dict(case=case, lib=lib, probs=probs, solver=solver)


def _run_batch(s):
    lib = s["lib"]
    for q in s["probs"]:
        q["T"].set_values(q["zero"])
    s["solver"].solve([q["eqn"] for q in s["probs"]])
    for q in s["probs"]:
        lib.check(lib.scalar_get_values(q["T"].h, _ptr(q["out"])))
    return [q["out"] for q in s["probs"]]


def _exact_batch(case, seed):
    """Each seven-point system in 64 bits by conjugate gradients, restarted from its true
    residual until that stops falling."""
    out = []
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    for N, kappa, f in _batch_coefficients(case, seed):
        h = 1.0 / N
        k = torch.from_numpy(kappa).to(dev).reshape(N, N, N)
        b = torch.from_numpy(f).to(dev).reshape(N, N, N) * h ** 3
        lo = [tuple(slice(0, N - 1) if d == a else slice(None) for d in range(3)) for a in range(3)]
        hi = [tuple(slice(1, N) if d == a else slice(None) for d in range(3)) for a in range(3)]
        g = [0.5 * h * (k[lo[a]] + k[hi[a]]) for a in range(3)]
        diag = torch.zeros_like(k)
        for a in range(3):
            diag[lo[a]] += g[a]
            diag[hi[a]] += g[a]
            for end in (0, N - 1):
                wall = tuple(end if d == a else slice(None) for d in range(3))
                diag[wall] += 2.0 * h * k[wall]

        def apply(x):
            y = diag * x
            for a in range(3):
                y[lo[a]] -= g[a] * x[hi[a]]
                y[hi[a]] -= g[a] * x[lo[a]]
            return y

        def dot(u, v):
            return float((u * v).sum())

        x, last = torch.zeros_like(b), np.inf
        for _ in range(4):
            r = b - apply(x)
            size = dot(r, r) ** 0.5
            if not size < 0.5 * last:
                break
            last, stop = size, 1e-8 * size
            z = r / diag
            p, rz = z, dot(r, z)
            while dot(r, r) ** 0.5 > stop:
                q = apply(p)
                alpha = rz / dot(p, q)
                x = x + alpha * p
                r = r - alpha * q
                z = r / diag
                rz, old = dot(r, z), rz
                p = z + (rz / old) * p
        out.append(x.reshape(-1).cpu().numpy())
    return out


# ---------------------------------------------------------------- adjoint on tetrahedra
def _prepare_adjoint(case, seed):
    lib = prism_b200.lib()
    rng = np.random.default_rng(seed)
    n = case["n"]
    mesh = api.Mesh(meshgen.box_tet(n, n, n), _box({"T": {p: ("fixed", 0.0) for p in WALLS}}), lib=lib)
    nc, nb = mesh.n_cells, mesh.info.n_boundary_faces
    kappa0 = rng.lognormal(0.0, 0.5, nc)
    fv = np.zeros(mesh.n_faces)
    fv[:nb] = rng.uniform(0.0, 1.0, nb)
    target = rng.normal(0.0, 1.0, nc)
    T = api.Scalar("T", mesh, 0.0)
    T.set_face_values(fv)
    kappa = api.Scalar("kappa", mesh, kappa0)
    eqn = api.Transport(api.diffusion.Corrected(kappa, T))
    return dict(case=case, lib=lib, mesh=mesh, T=T, kappa=kappa, eqn=eqn, kappa0=_pinned(kappa0), fv=_pinned(fv),
                target=target, vol=mesh.export()["cell_volume"], zero=_pinned(np.zeros(nc)),
                phi=_pinned(np.zeros(nc)), solver=api.BiCGSTAB(krylov_tol=1e-13, krylov_max_iter=100000))


def _run_adjoint(s):
    lib = s["lib"]
    s["kappa"].set_values(s["kappa0"])
    s["T"].set_values(s["zero"])
    s["T"].set_face_values(s["fv"])
    api.adjoint_forward(s["eqn"], s["solver"], max_outer=200, outer_tol=1e-12)
    lib.check(lib.scalar_get_values(s["T"].h, _ptr(s["phi"])))
    dJ = 2.0 * s["vol"] * (s["phi"] - s["target"])
    gk, gv, _ = api.adjoint_backward(s["eqn"], dJ, s["solver"], max_outer=200, outer_tol=1e-12)
    return {"phi": s["phi"], "dJ_dkappa": gk, "dJ_dv": gv}


# ---------------------------------------------------------------- the interface
_PREPARE = {"poisson": _prepare_poisson, "simple": _prepare_simple, "transport": _prepare_transport,
            "transient": _prepare_transient, "batch": _prepare_batch, "adjoint": _prepare_adjoint}
_RUN = {"poisson": _run_poisson, "simple": _run_simple, "transport": _run_transport, "transient": _run_transient,
        "batch": _run_batch, "adjoint": _run_adjoint}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["case"]["kind"]](state)


def exact(case, seed):
    if case["kind"] == "poisson":
        return _exact_poisson(case, seed)
    if case["kind"] == "batch":
        return _exact_batch(case, seed)
    return None


def work(case):
    """Each system's matrix (FP64 values and 32-bit columns), right-hand side, solution and the
    face and cell geometry it is assembled from, read or written once per assembled solve."""
    kind = case["kind"]

    def system(cells, faces, row):
        return cells * (row * 12 + 4 + 2 * 8 + 4 * 8) + faces * 10 * 8

    if kind in ("poisson", "transport", "simple"):
        cells = case["nx"] * case["ny"] * case["nz"]
        flat = case["nz"] == 1
        one = system(cells, (2 if flat else 3) * cells, 5 if flat else 7)
        row = 5 if flat else 7
        solves = case["steps"] * ((2 if flat else 3) + 3) if kind == "simple" else 1
    elif kind == "batch":
        cells = sum(N ** 3 for N in _batch_sizes(case))
        one, row, solves = system(cells, 3 * cells, 7), 7, 1
    else:
        cells = 6 * case["n"] ** 3
        one, row = system(cells, 2 * cells, 5), 5
        solves = 2 * case["steps"] if kind == "transient" else 2
    return {"bytes": float(one * solves), "flops": float(2 * row * cells * solves)}
