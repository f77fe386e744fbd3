"""The work a user of cloudfem_b200 has it do, as cases that can be timed.

``listed()`` names them, ``draw(rng)`` gives another case of the same ranges,
``prepare`` makes what a program has in hand before the call, ``run`` is one
pass through the public entry points, ``exact`` the same answer in plain
64-bit torch, ``work`` the bytes and operations one pass cannot do without.

Kinds and their ranges (cells per box edge; a cell is six tetrahedra):

* ``p1_poisson``   ``solve_tet_poisson``: P1 heat, from a few hundred nodes
  (a call's latency) over the 20^3 manufactured problem to 48^3 cells
* ``t10_poisson``  ``solve_tet10_poisson``: Tet10 heat, up to 24^3 cells
* ``t10_assemble`` ``assemble_tet10``: stiffness and load as SciPy CSR
* ``t10_elastic``  ``solve_elasticity_tet10``: clamped box under a face
  traction, cantilevers and blocks, up to 5,300 cells
* ``p1_elastic``   ``solve_elasticity_3d`` and ``element_stress_strain_3d``:
  weight and a temperature field, stresses recovered from the displacement
* ``p1_march``     ``transient_heat_tet``: Crank-Nicolson with convection on
  every face and a Gaussian source
* ``batch``        ``solve_batch``: independent Tet10 meshes of 4 to 24 cells
  per edge with a lognormal conductivity per cell, meshes resident
* ``resident``     a design loop on one large resident mesh: reassemble with
  new coefficients, refresh the solve plan, solve, all on the device
* ``phasor``       ``solve_eddy_current_tet10`` in a conductor
* ``serve``        ``Server.serve``: a mixed stream on resident meshes
"""

import functools
import math

import numpy as np
import torch

from cloudfem_b200 import _native as N
from cloudfem_b200 import serve
from cloudfem_b200.batch import BatchSolver, HeatProblem, solve_batch
from cloudfem_b200.device import BlockSystem, DeviceMesh, PcgPlan, fixed_mask, fixed_scalar
from cloudfem_b200.fem.tet10 import assemble_tet10, solve_tet10_poisson
from cloudfem_b200.fem.tet_heat import transient_heat_tet
from cloudfem_b200.fem.tet_poisson import solve_tet_poisson
from cloudfem_b200.mesh import Tet10Mesh, TetMesh, box_mesh, box_mesh_tet10
from cloudfem_b200.physics.elastic3d import element_stress_strain_3d, solve_elasticity_3d
from cloudfem_b200.physics.elastic_tet10 import solve_elasticity_tet10
from cloudfem_b200.physics.em3d_tet10 import solve_eddy_current_tet10

FACES = ("xmin", "xmax", "ymin", "ymax", "zmin", "zmax")
ZERO_BC = {s: 0.0 for s in FACES}


def listed():
    return [
        # a tiny model: what a call costs before any arithmetic
        {"name": "p1 poisson 6x5x4", "kind": "p1_poisson", "nx": 6, "ny": 5, "nz": 4, "precision": "fp64"},
        # the plain steady heat problem of the test suite
        {"name": "p1 poisson 20x20x20", "kind": "p1_poisson", "nx": 20, "ny": 20, "nz": 20, "precision": "fp64"},
        # an ordinary quadratic heat model, ragged, mixed precision
        {"name": "t10 poisson 23x17x13", "kind": "t10_poisson", "nx": 23, "ny": 17, "nz": 13, "precision": "mixed"},
        # a caller that takes the assembled system to its own SciPy code
        {"name": "t10 assemble 17x16x15", "kind": "t10_assemble", "nx": 17, "ny": 16, "nz": 15},
        # a bending cantilever, plain FP64: many iterations on a small system
        {"name": "t10 elastic 40x5x5", "kind": "t10_elastic", "nx": 40, "ny": 5, "nz": 5, "precision": "fp64"},
        # a block under traction, mixed precision: past one resident wave
        {"name": "t10 elastic 27x15x13", "kind": "t10_elastic", "nx": 27, "ny": 15, "nz": 13, "precision": "mixed"},
        # a linear part under weight and heat, with its stresses
        {"name": "p1 elastic 31x17x14", "kind": "p1_elastic", "nx": 31, "ny": 17, "nz": 14, "precision": "fp64"},
        # a cooling part over time: short warm-started solves
        {"name": "p1 march 40x36x33", "kind": "p1_march", "nx": 40, "ny": 36, "nz": 33, "steps": 20,
         "precision": "mixed"},
        # many small meshes at once (parameter studies)
        {"name": "batch of 48", "kind": "batch", "meshes": 48, "nmin": 4, "nmax": 24, "mix": 0,
         "precision": "mixed"},
        # one large mesh kept on the device, new coefficients each pass
        {"name": "resident 96x88x80", "kind": "resident", "nx": 96, "ny": 88, "nz": 80},
        # an eddy-current phasor solve
        {"name": "phasor 7x6x6", "kind": "phasor", "nx": 7, "ny": 6, "nz": 6},
        # a served stream of small and middling requests
        {"name": "serve 24", "kind": "serve", "requests": 24, "dmin": 1000, "dmax": 60000, "mix": 0},
    ]


# cells per edge of a drawn case (smallest, largest) and, above, the most
# cells in all; each kind's largest is no more than its listed one costs
RANGES = {"p1_poisson": (4, 48, 48 ** 3), "t10_poisson": (3, 24, 24 ** 3),
          "t10_assemble": (3, 20, 20 ** 3), "t10_elastic": (3, 30, 5300),
          "p1_elastic": (4, 32, 7400), "p1_march": (6, 40, 47500),
          "resident": (24, 96, 96 * 88 * 80), "phasor": (3, 7, 252)}


def draw(rng):
    kind = rng.choice(["p1_poisson", "t10_poisson", "t10_assemble", "t10_elastic", "p1_elastic",
                       "p1_march", "batch", "resident", "phasor", "serve"])
    if kind == "batch":
        nmin = rng.randint(3, 8)
        return {"kind": kind, "meshes": rng.randint(2, 48), "nmin": nmin,
                "nmax": rng.randint(nmin + 2, 24), "mix": rng.randint(1, 10 ** 6),
                "precision": rng.choice(["mixed", "fp64"])}
    if kind == "serve":
        dmin = int(round(math.exp(rng.uniform(math.log(1e3), math.log(8e3)))))
        return {"kind": kind, "requests": rng.randint(3, 24), "dmin": dmin,
                "dmax": int(round(dmin * math.exp(rng.uniform(1.0, 2.0)))),
                "mix": rng.randint(1, 10 ** 6)}
    lo, hi, most = RANGES[kind]
    while True:
        e = [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(3)]
        if e[0] * e[1] * e[2] <= most:
            break
    if kind == "t10_elastic":
        e = sorted(e, reverse=True)      # clamped at the end of the long axis
        e[0] = min(e[0], 5 * e[1])
    c = {"kind": kind, "nx": e[0], "ny": e[1], "nz": e[2]}
    if kind in ("p1_poisson", "t10_poisson", "t10_elastic", "p1_elastic"):
        c["precision"] = rng.choice(["fp64", "mixed"])
    if kind == "p1_march":
        c["steps"] = rng.randint(4, 20)
        c["precision"] = rng.choice(["fp64", "mixed"])
    return c


# ------------------------------------------------------------------ meshes

@functools.lru_cache(maxsize=96)
def _box(nx, ny, nz, tet10):
    return (box_mesh_tet10 if tet10 else box_mesh)(nx, ny, nz)


def _mesh(nx, ny, nz, tet10, lims):
    """The box [0, lims], on connectivity that is made once per grid."""
    m = _box(nx, ny, nz, tet10)
    nodes = m.nodes * np.asarray(lims, dtype=float)
    if tet10:
        return Tet10Mesh(nodes, m.elements, m.boundaries, n_corners=m.n_corners)
    return TetMesh(nodes, m.elements, m.boundaries)


def _case_mesh(case, rng):
    tet10 = case["kind"] in ("t10_poisson", "t10_assemble", "t10_elastic", "phasor")
    lims = rng.uniform(0.8, 1.2, 3)
    if case["kind"] in ("t10_elastic", "p1_elastic"):   # cubic cells, a part in metres
        lims = lims * np.array([case["nx"], case["ny"], case["nz"]]) / (40.0 * 1.25)
    return _mesh(case["nx"], case["ny"], case["nz"], tet10, lims)


def _fields(rng):
    """A smooth conductivity and source, as callables of the coordinates."""
    a, b, c, p, q = rng.uniform(0.2, 0.8, 5)

    def k(x, y, z):
        return 1.0 + a * np.sin(3.0 * x + p) * np.cos(2.0 * y) + b * z * z

    def f(x, y, z):
        return np.sin(np.pi * x) * np.sin(np.pi * y + q) + c * z

    return k, f


def _batch_cells(case):
    return np.random.default_rng(case["mix"]).integers(case["nmin"], case["nmax"] + 1,
                                                       case["meshes"]).tolist()


def _requests(case):
    """Kind and cells of every request of a stream (sizes log-uniform)."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["requests"]):
        kind = ("p1_heat", "t10_heat", "t10_elast")[int(rng.choice(3, p=(0.6, 0.25, 0.15)))]
        dofs = math.exp(rng.uniform(math.log(case["dmin"]), math.log(case["dmax"])))
        cells = max(dofs / {"p1_heat": 1.0, "t10_heat": 8.0, "t10_elast": 24.0}[kind], 8.0)
        aspect = rng.uniform(1.0, 4.0)
        ny = max(1, int(round((cells / aspect) ** (1.0 / 3.0))))
        out.append((kind, max(1, int(round(aspect * ny))), ny, ny))
    return out


# ------------------------------------------------------------------- cases

def _inputs(case, seed):
    """Host inputs of a case, from its seed alone."""
    rng = np.random.default_rng([int(seed), 17])
    kind = case["kind"]
    if kind == "batch":
        return [(_mesh(n, n, n, True, (1.0, 1.0, 1.0)), np.repeat(rng.lognormal(0.0, 1.0, n ** 3), 6))
                for n in _batch_cells(case)]
    if kind == "serve":
        out = []
        for rk, nx, ny, nz in _requests(case):
            m = _mesh(nx, ny, nz, rk != "p1_heat", (nx / ny, 1.0, 1.0))
            coef = (210e9 * rng.lognormal(0.0, 0.5) if rk == "t10_elast"
                    else np.repeat(rng.lognormal(0.0, 0.5, nx * ny * nz), 6))
            out.append((rk, m, coef))
        return out
    s = {"mesh": _case_mesh(case, rng)}
    if kind in ("p1_poisson", "t10_poisson", "t10_assemble"):
        s["k"], s["f"] = _fields(rng)
        s["bc"] = dict(ZERO_BC, xmin=float(rng.uniform(0.5, 1.5)))
    elif kind == "t10_elastic":
        s["E"], s["nu"] = 210e9 * rng.uniform(0.8, 1.2), 0.3
        s["traction"] = {"xmax": (float(rng.uniform(0.0, 1e6)), 0.0, -1e6)}
    elif kind == "p1_elastic":
        s["E"], s["nu"] = 70e9 * rng.uniform(0.8, 1.2), 0.33
        s["body"] = (0.0, 0.0, -2700.0 * 9.81 * float(rng.uniform(0.9, 1.1)))
        x = s["mesh"].nodes
        s["T"] = 20.0 + 60.0 * rng.uniform(0.5, 1.5) * x[:, 0] * x[:, 2]
        s["alpha"], s["T_ref"] = 23e-6, 20.0
    elif kind == "p1_march":
        s["h"], s["peak"] = 25.0 * rng.uniform(0.5, 2.0), 1e7 * rng.uniform(0.5, 1.5)
    elif kind == "resident":
        s["k"] = rng.lognormal(0.0, 0.5, len(s["mesh"].elements) // 6).repeat(6)
    elif kind == "phasor":
        s["B"] = (0.0, float(rng.uniform(0.0, 0.5)), 1.0)
        s["sigma"] = 1e6 * rng.uniform(0.8, 1.2)
    return s


def _gauss(peak):
    def f(x, y, z):
        return peak * np.exp(-((x - 0.5) ** 2 + (y - 0.5) ** 2 + (z - 0.5) ** 2) / (2.0 * 0.1 ** 2))
    return f


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        solver = BatchSolver()
        for m, _ in s:
            solver.device_mesh(m)
        return {"case": case, "solver": solver,
                "problems": [HeatProblem(m, k=k, f=1.0, bc=ZERO_BC) for m, k in s]}
    if kind == "serve":
        return {"case": case, "server": serve.Server(), "requests": s}
    s["case"] = case
    if kind == "resident":
        dm = DeviceMesh(s["mesh"])
        pat = dm.pattern
        n = dm.n_nodes
        dev = dm.nodes.device
        idx, val = fixed_scalar(s["mesh"], ZERO_BC)
        mask, x0 = fixed_mask(dm.rt, n, idx, val)
        vals = torch.zeros(pat.nnz, dtype=torch.float64, device=dev)
        rhs = torch.zeros(n, dtype=torch.float64, device=dev)
        dm.assemble(N.OP_P1_STIFF, coef=1.0, load=1.0, vals=vals, rhs=rhs)
        system = BlockSystem(dm.rt, n, 1, pat.row_ptr, pat.col, vals, rhs, x0.clone(), mask)
        s.update(dm=dm, x0=x0, vals=vals, rhs=rhs, system=system,
                 plan=PcgPlan([system], N.SOLVE_FP64, 1e-12))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "p1_poisson":
        return solve_tet_poisson(s["mesh"], k=s["k"], f=s["f"], bc=s["bc"], precision=case["precision"])
    if kind == "t10_poisson":
        return solve_tet10_poisson(s["mesh"], k=s["k"], f=s["f"], bc=s["bc"], precision=case["precision"])
    if kind == "t10_assemble":
        A, rhs = assemble_tet10(s["mesh"], k=s["k"], f=s["f"])
        return {"data": A.data, "indices": A.indices, "indptr": A.indptr, "rhs": rhs}
    if kind == "t10_elastic":
        return np.stack(solve_elasticity_tet10(s["mesh"], s["E"], s["nu"], bc={"xmin": (0.0, 0.0, 0.0)},
                                               traction=s["traction"], precision=case["precision"]))
    if kind == "p1_elastic":
        u = solve_elasticity_3d(s["mesh"], s["E"], s["nu"], bc={"xmin": (0.0, 0.0, 0.0)}, body=s["body"],
                                T=s["T"], alpha=s["alpha"], T_ref=s["T_ref"], precision=case["precision"])
        sig, eps = element_stress_strain_3d(s["mesh"], u, s["E"], s["nu"], T=s["T"], alpha=s["alpha"],
                                            T_ref=s["T_ref"])
        return {"u": np.stack(u), "sig": sig, "eps": eps}
    if kind == "p1_march":
        return transient_heat_tet(s["mesh"], k=45.0, rho_cp=3.6e6, f=_gauss(s["peak"]),
                                  robin={n: (s["h"], 20.0) for n in FACES}, t_end=float(case["steps"]),
                                  dt=1.0, T0=20.0, method="cn", precision=case["precision"])[1]
    if kind == "batch":
        return solve_batch(s["problems"], precision=case["precision"], solver=s["solver"])
    if kind == "resident":
        s["dm"].assemble(N.OP_P1_STIFF, coef=s["k"], load=1.0, vals=s["vals"], rhs=s["rhs"])
        s["plan"].refresh()
        s["system"].x.copy_(s["x0"])
        s["plan"].solve()
        return s["system"].x
    if kind == "phasor":
        a, v = solve_eddy_current_tet10(s["mesh"], sigma=s["sigma"], omega=2.0 * np.pi * 1000.0,
                                        B_applied=s["B"])
        return {"a": a, "v": v}
    reqs = [serve.Request(i, rk, m, **({"E": c} if rk == "t10_elast" else {"k": c}))
            for i, (rk, m, c) in enumerate(s["requests"])]
    s["server"].serve(reqs, realtime=False)
    return [r.result for r in reqs]


# -------------------------------------------------------------------- work

def _sizes(nx, ny, nz, tet10):
    """(nodes, elements, stored entries of the node pattern)."""
    n, m = (nx + 1) * (ny + 1) * (nz + 1), 6 * nx * ny * nz
    if not tet10:
        return n, m, 15 * n
    return (2 * nx + 1) * (2 * ny + 1) * (2 * nz + 1), m, 8 * 28 * nx * ny * nz


def _one(nx, ny, nz, tet10, comp, solve=True):
    """Mesh in, solution out; element matrices and one product with the
    matrix are the least any solve takes."""
    n, m, nnz = _sizes(nx, ny, nz, tet10)
    npe = 10 if tet10 else 4
    b = 24 * n + 4 * npe * m + 8 * comp * n
    fl = m * (5 * npe * npe * 6 * comp * comp if tet10 else 16 * 6 * comp * comp)
    if solve:
        b += nnz * (8 * comp * comp + 4)
        fl += 2 * nnz * comp * comp
    return b, fl


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [_one(n, n, n, True, 1) for n in _batch_cells(case)]
    elif kind == "serve":
        parts = [_one(nx, ny, nz, rk != "p1_heat", 3 if rk == "t10_elast" else 1)
                 for rk, nx, ny, nz in _requests(case)]
    else:
        e = (case["nx"], case["ny"], case["nz"])
        tet10 = kind in ("t10_poisson", "t10_assemble", "t10_elastic", "phasor")
        comp = 3 if kind in ("t10_elastic", "p1_elastic", "phasor") else 1
        parts = [_one(*e, tet10, comp, kind != "t10_assemble")]
        n, m, nnz = _sizes(*e, tet10)
        if kind == "t10_assemble":
            parts.append((12 * nnz + 12 * n, 0))
        if kind == "p1_elastic":
            parts.append((2 * 48 * m, 100 * m))
        if kind == "p1_march":     # every step: both matrices once, the field out
            parts.append((case["steps"] * (nnz * 20 + 8 * n), case["steps"] * 4 * nnz))
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


# ------------------------------------------------------------------- exact

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=_dev())


_EDGES = ((0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3))


def _rule(npe):
    """(weights (Q,), N (Q, npe), dN/dxi (Q, npe, 3)) of the element rule."""
    a, b = 0.5, 1.0 / 6.0
    if npe == 4:
        L, w = np.full((1, 4), 0.25), np.array([1.0])
    else:
        L = np.array([[0.25] * 4, [a, b, b, b], [b, a, b, b], [b, b, a, b], [b, b, b, a]])
        w = np.array([-0.8, 0.45, 0.45, 0.45, 0.45])
    q = len(w)
    Nv, dN = np.zeros((q, npe)), np.zeros((q, npe, 4))
    for i in range(4):
        Nv[:, i] = L[:, i] if npe == 4 else L[:, i] * (2.0 * L[:, i] - 1.0)
        dN[:, i, i] = 1.0 if npe == 4 else 4.0 * L[:, i] - 1.0
    if npe == 10:
        for e, (i, j) in enumerate(_EDGES):
            Nv[:, 4 + e] = 4.0 * L[:, i] * L[:, j]
            dN[:, 4 + e, i], dN[:, 4 + e, j] = 4.0 * L[:, j], 4.0 * L[:, i]
    dxi = np.stack([dN[..., k] - dN[..., 0] for k in (1, 2, 3)], axis=-1)
    return _t(w), _t(Nv), _t(dxi), L


def _geometry(mesh):
    """(elements, volumes, G (M, Q, npe, 3), weights, N, points (M, Q, 3))."""
    x, els = _t(mesh.nodes), _t(mesh.elements)
    w, Nv, dxi, L = _rule(els.shape[1])
    p = x[els[:, :4]]
    J = torch.stack([p[:, c] - p[:, 0] for c in (1, 2, 3)], dim=2)
    vol = torch.linalg.det(J).abs() / 6.0
    G = torch.einsum("qpk,ekl->eqpl", dxi, torch.linalg.inv(J))
    return els, vol, G, w, Nv, torch.einsum("qc,ecx->eqx", _t(L), p)


def _at(spec, pts, m):
    """Values (M, Q) of a number, a per-element array or a callable."""
    q = pts.shape[1]
    if callable(spec):
        h = pts.reshape(-1, 3).cpu().numpy()
        return _t(spec(h[:, 0], h[:, 1], h[:, 2])).reshape(m, q)
    if isinstance(spec, np.ndarray):
        return _t(spec)[:, None].expand(m, q)
    return torch.full((m, q), float(spec), dtype=torch.float64, device=_dev())


def _csr(rows, cols, vals, shape):
    idx = torch.stack([rows.reshape(-1), cols.reshape(-1)])
    return torch.sparse_coo_tensor(idx, vals.reshape(-1), shape).coalesce().to_sparse_csr()


def _scalar(mesh, k, f):
    """Stiffness (CSR) and load of -div(k grad u) = f."""
    els, vol, G, w, Nv, pts = _geometry(mesh)
    m, npe = els.shape
    kq = _at(k, pts, m) * w * vol[:, None]
    ke = torch.einsum("eq,eqax,eqbx->eab", kq, G, G)
    n = mesh.n_nodes
    A = _csr(els[:, :, None].expand(m, npe, npe), els[:, None, :].expand(m, npe, npe), ke, (n, n))
    fe = torch.einsum("eq,qa->ea", _at(f, pts, m) * w * vol[:, None], Nv)
    b = torch.zeros(n, dtype=torch.float64, device=_dev()).index_add_(0, els.reshape(-1), fe.reshape(-1))
    return A, b


def _blocks(els, ke, n, comp=3):
    """CSR over DOFs 3 p + c from element blocks (M, npe, npe, 3, 3)."""
    d = 3 * els[:, :, None] + torch.arange(3, device=els.device)
    m, npe = els.shape
    shape = (m, npe, npe, 3, 3)
    rows = d[:, :, None, :, None].expand(shape)
    cols = d[:, None, :, None, :].expand(shape)
    return _csr(rows, cols, ke, (comp * n, comp * n))


def _elastic(mesh, E, nu, body=None, T=None, alpha=0.0, T_ref=0.0):
    els, vol, G, w, Nv, _ = _geometry(mesh)
    lam, mu = E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu)), E / (2.0 * (1.0 + nu))
    wv = w * vol[:, None]
    outer = torch.einsum("eq,eqac,eqbd->eabcd", wv, G, G)
    dot = torch.einsum("eabcc->eab", outer)
    ke = lam * outer + mu * outer.transpose(3, 4)
    ke = ke + mu * dot[..., None, None] * torch.eye(3, dtype=torch.float64, device=_dev())
    n = mesh.n_nodes
    fe = torch.zeros(els.shape + (3,), dtype=torch.float64, device=_dev())
    if body is not None:
        fe += torch.einsum("eq,qa->ea", wv, Nv)[..., None] * _t(np.array(body))
    if T is not None:
        th = (3.0 * lam + 2.0 * mu) * alpha * (torch.einsum("qa,ea->eq", Nv, _t(T)[els]) - T_ref)
        fe += torch.einsum("eq,eqac->eac", wv * th, G)
    b = torch.zeros(3 * n, dtype=torch.float64, device=_dev())
    b.index_add_(0, (3 * els[..., None] + torch.arange(3, device=els.device)).reshape(-1), fe.reshape(-1))
    return _blocks(els, ke, n), b


def _named_faces(mesh, name):
    """Corner triples (and the element's local indexes) on a flat side."""
    inset = np.zeros(mesh.n_nodes, dtype=bool)
    inset[np.asarray(mesh.boundaries[name])] = True
    els = np.asarray(mesh.elements)
    tri = ((0, 1, 2), (0, 1, 3), (0, 2, 3), (1, 2, 3))
    out = []
    for t in tri:
        sel = inset[els[:, t]].all(axis=1)
        nodes = els[sel][:, t]
        if els.shape[1] == 10:
            mid = [4 + [set(e) for e in _EDGES].index({t[i], t[j]}) for i, j in ((0, 1), (1, 2), (2, 0))]
            nodes = np.concatenate([nodes, els[sel][:, mid]], axis=1)
        out.append(nodes)
    f = np.concatenate(out)
    p = mesh.nodes[f[:, :3]]
    return f, 0.5 * np.linalg.norm(np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]), axis=1)


def _cg(A, b, free, x, rounds=3, most=40000):
    """Jacobi CG with refinement on the free unknowns; x holds the fixed."""
    free = free.to(torch.float64)
    n = b.numel()
    rows = torch.repeat_interleave(torch.arange(n, device=b.device), A.crow_indices().diff())
    on = rows == A.col_indices()
    dinv = torch.zeros_like(b)
    dinv[rows[on]] = free[rows[on]] / A.values()[on]
    for _ in range(rounds):
        r = (b - A @ x) * free
        z = dinv * r
        p, d = z.clone(), torch.zeros_like(x)
        rz = torch.dot(r, z)
        stop = float(rz) * 1e-26
        for it in range(most):
            if it % 32 == 0 and not float(rz) > stop:
                break
            q = (A @ p) * free
            a = rz / torch.dot(p, q)
            d += a * p
            r -= a * q
            z = dinv * r
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
        x = x + d
    return x


def _fixed(n, parts):
    """(free mask, x) on the device from [(indices, values)]."""
    free = torch.ones(n, dtype=torch.bool, device=_dev())
    x = torch.zeros(n, dtype=torch.float64, device=_dev())
    for idx, val in parts:
        i = _t(np.asarray(idx, dtype=np.int64))
        free[i] = False
        x[i] = val
    return free, x


def _heat(mesh, k, f, bc):
    A, b = _scalar(mesh, k, f)
    free, x = _fixed(mesh.n_nodes, [(mesh.boundaries[s], v) for s, v in bc.items()])
    return _cg(A, b, free, x)


def _clamped(mesh, E, nu, traction):
    A, b = _elastic(mesh, E, nu)
    for name, t in traction.items():
        faces, area = _named_faces(mesh, name)
        # a constant traction on a straight quadratic face: a third of it on each midside node
        add = _t(area)[:, None, None] / 3.0 * _t(np.array(t)) * torch.ones((1, 3, 1), device=_dev(),
                                                                            dtype=torch.float64)
        d = 3 * _t(faces[:, 3:])[..., None] + torch.arange(3, device=_dev())
        b.index_add_(0, d.reshape(-1), add.reshape(-1))
    free, x = _fixed(3 * mesh.n_nodes, [(3 * np.asarray(mesh.boundaries["xmin"]) + c, 0.0) for c in range(3)])
    return _cg(A, b, free, x)


def _mass(mesh, rho):
    """Consistent capacity matrix as element blocks (M, npe, npe)."""
    els, vol, _, _, _, _ = _geometry(mesh)
    npe = els.shape[1]
    if npe == 4:
        ref = (np.ones((4, 4)) + np.eye(4)) / 20.0
    else:
        ref = np.zeros((10, 10))
        ref[:4, :4] = np.ones((4, 4)) + 5.0 * np.eye(4)
        for e, (i, j) in enumerate(_EDGES):
            for c in range(4):
                ref[c, 4 + e] = ref[4 + e, c] = -4.0 if c in (i, j) else -6.0
            for g, o in enumerate(_EDGES):
                ref[4 + e, 4 + g] = {0: 8.0, 1: 16.0, 2: 32.0}[len({i, j} & set(o))]
        ref /= 420.0
    return els, rho * vol[:, None, None] * _t(ref)


def _march(s, case):
    mesh = s["mesh"]
    n = mesh.n_nodes
    K, F = _scalar(mesh, 45.0, _gauss(s["peak"]))
    K = K.to_sparse_coo()
    els, ce = _mass(mesh, 3.6e6)
    m = els.shape[0]
    C = _csr(els[:, :, None].expand(m, 4, 4), els[:, None, :].expand(m, 4, 4), ce, (n, n)).to_sparse_coo()
    for name in FACES:
        f, area = _named_faces(mesh, name)
        f, area = _t(f), _t(area)
        he = s["h"] * area[:, None, None] / 12.0 * (1.0 + torch.eye(3, dtype=torch.float64, device=_dev()))
        K = K + _csr(f[:, :, None].expand(len(f), 3, 3), f[:, None, :].expand(len(f), 3, 3), he,
                     (n, n)).to_sparse_coo()
        F.index_add_(0, f.reshape(-1), (s["h"] * 20.0 * area / 3.0)[:, None].expand(len(f), 3).reshape(-1))
    L, R = ((C + w * K).coalesce().to_sparse_csr() for w in (0.5, -0.5))
    T = torch.full((n,), 20.0, dtype=torch.float64, device=_dev())
    free = torch.ones(n, dtype=torch.bool, device=_dev())
    out = [T]
    for _ in range(case["steps"]):
        T = _cg(L, R @ T + F, free, T, rounds=2)
        out.append(T)
    return torch.stack(out)


def _phasor(s):
    """COCG on the reduced system, the V rows scaled by 1 / (i omega)."""
    mesh, sig, w_ = s["mesh"], s["sigma"], 2.0 * np.pi * 1000.0
    els, vol, G, w, Nv, _ = _geometry(mesh)
    n = mesh.n_nodes
    wv = w * vol[:, None]
    nu = 1.0 / (4e-7 * np.pi)
    outer = torch.einsum("eq,eqac,eqbd->eabcd", wv, G, G)
    eye = torch.eye(3, dtype=torch.float64, device=_dev())
    ke = nu * (torch.einsum("eabcc->eab", outer)[..., None, None] * eye - outer.transpose(3, 4))
    _, me = _mass(mesh, sig)
    ae = torch.complex(ke, w_ * me[..., None, None] * eye)
    m = els.shape[0]
    # unknowns 4 p + (Ax, Ay, Az, V); the V block is grad-grad / (i omega)
    full = torch.zeros((m, 10, 10, 4, 4), dtype=torch.complex128, device=_dev())
    full[..., :3, :3] = ae
    ge = sig * torch.einsum("eq,qa,eqbc->eabc", wv, Nv, G)
    full[..., :3, 3] = ge.to(torch.complex128)
    full[..., 3, :3] = ge.transpose(1, 2).to(torch.complex128)
    full[..., 3, 3] = sig * torch.einsum("eabcc->eab", outer) / (1j * w_)
    d = 4 * els[:, :, None] + torch.arange(4, device=els.device)
    shape = (m, 10, 10, 4, 4)
    A = _csr(d[:, :, None, :, None].expand(shape), d[:, None, :, None, :].expand(shape), full, (4 * n, 4 * n))
    x = torch.zeros(4 * n, dtype=torch.complex128, device=_dev())
    free = torch.ones(4 * n, dtype=torch.bool, device=_dev())
    bnd = np.unique(np.concatenate([np.asarray(mesh.boundaries[f]) for f in FACES]))
    val = _t(0.5 * np.cross(np.array(s["B"]), mesh.nodes[bnd])).to(torch.complex128)
    for c in range(3):
        x[_t(4 * bnd + c)] = val[:, c]
        free[_t(4 * bnd + c)] = False
    free[3] = False                    # V is pinned at the first node
    fm = free.to(torch.complex128)
    rows = torch.repeat_interleave(torch.arange(4 * n, device=_dev()), A.crow_indices().diff())
    on = rows == A.col_indices()
    dinv = torch.zeros_like(x)
    dinv[rows[on]] = fm[rows[on]] / A.values()[on]
    for _ in range(2):
        r = -(A @ x) * fm
        z = dinv * r
        p, dx, rz = z.clone(), torch.zeros_like(x), (r * z).sum()
        stop = 1e-13 * float(r.abs().square().sum().sqrt())
        for it in range(30000):
            if it % 64 == 0 and not float(r.abs().square().sum().sqrt()) > stop:
                break
            q = (A @ p) * fm
            a = rz / (p * q).sum()
            dx += a * p
            r -= a * q
            z = dinv * r
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
        x = x + dx
    x = x.reshape(n, 4)
    return {"a": x[:, :3].reshape(-1), "v": x[:, 3].contiguous()}


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind in ("p1_poisson", "t10_poisson"):
        return _heat(s["mesh"], s["k"], s["f"], s["bc"])
    if kind == "t10_assemble":
        A, rhs = _scalar(s["mesh"], s["k"], s["f"])
        return {"data": A.values(), "indices": None, "indptr": None, "rhs": rhs}
    if kind == "t10_elastic":
        return _clamped(s["mesh"], s["E"], s["nu"], s["traction"]).reshape(-1, 3).T.contiguous()
    if kind == "p1_elastic":
        mesh = s["mesh"]
        A, b = _elastic(mesh, s["E"], s["nu"], s["body"], s["T"], s["alpha"], s["T_ref"])
        free, x = _fixed(3 * mesh.n_nodes,
                         [(3 * np.asarray(mesh.boundaries["xmin"]) + c, 0.0) for c in range(3)])
        u = _cg(A, b, free, x).reshape(-1, 3)
        els, _, G, _, Nv, _ = _geometry(mesh)
        g = torch.einsum("eac,ead->ecd", G[:, 0], u[els])        # du_d / dx_c
        eps = torch.stack([g[:, 0, 0], g[:, 1, 1], g[:, 2, 2], g[:, 1, 2] + g[:, 2, 1],
                           g[:, 0, 2] + g[:, 2, 0], g[:, 0, 1] + g[:, 1, 0]], dim=1)
        E, nu = s["E"], s["nu"]
        lam, mu = E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu)), E / (2.0 * (1.0 + nu))
        th = s["alpha"] * ((_t(s["T"])[els] * Nv[0]).sum(dim=1) - s["T_ref"])
        em = eps.clone()
        em[:, :3] -= th[:, None]
        sig = mu * em
        sig[:, :3] = 2.0 * mu * em[:, :3] + lam * em[:, :3].sum(dim=1, keepdim=True)
        return {"u": u.T.contiguous(), "sig": sig, "eps": eps}
    if kind == "p1_march":
        return _march(s, case)
    if kind == "batch":
        return [_heat(m, k, 1.0, ZERO_BC) for m, k in s]
    if kind == "resident":
        return _heat(s["mesh"], s["k"], 1.0, ZERO_BC)
    if kind == "phasor":
        return _phasor(s)
    return [_clamped(m, c, 0.3, {"xmax": (0.0, 0.0, -1e6)}) if rk == "t10_elast"
            else _heat(m, c, 1.0, ZERO_BC) for rk, m, c in s]
