"""The calls a user of the library makes, as cases whose passes are timed and whose outputs are compared.

A case is a dict of plain values with a "kind" (below) and sizes.  prepare() builds what a program has in hand
before the call (mesh, model, numbered DOFs, boundary values, states), run() is one pass through the public entry
points, work() counts what the path cannot do without, and exact() restates the result in 64 bits with torch
and numpy alone, where the problem is one that a short program can solve.

Linear solves run to linear_rtol = 1e-10, the tolerance at which the tests compare solves: U and F are then given
to many digits, whatever the order of the solver's FP32 operations.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (_ROOT, os.path.join(_ROOT, "amaru.jl_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import amaru_gpu as A  # noqa: E402
from amaru_gpu import _lib as L  # noqa: E402
from amaru_gpu import serve, workloads  # noqa: E402

RTOL = 1e-10
_METHOD = {"mixed": L.SOLVER_MIXED, "amg": L.SOLVER_AMG}
_CELL = {"quad4": L.QUAD4, "quad8": L.QUAD8, "tet10": L.TET10, "hex8": L.HEX8, "hex20": L.HEX20}
_NEN = {"quad4": 4, "quad8": 8, "tet10": 10, "hex8": 8, "hex20": 20}
_NIP = {"quad4": 4, "quad8": 9, "tet10": 4, "hex8": 8, "hex20": 27}  # integration points the cases use


# ---------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest analysis of the benchmark, through MechAnalysis.solve with the default solver: DOF numbering,
        # load assembly, one Newton increment of 1 575 DOFs; latency and launches
        dict(name="cantilever_hex8_20x4x4", kind="analysis", cell="hex8", nx=20, ny=4, nz=4),
        # an elastoplastic plane-stress beam bent by a prescribed end displacement, default solver, Newton iterations
        # and the return mapping on a mesh of odd sizes
        dict(name="beam_vm_quad8_61x7", kind="beam", cell="quad8", nx=61, ny=7, nincs=6),
        # an ordinary linear stage: 37 000 DOFs with the multigrid solver
        dict(name="block_hex20_25x11x11", kind="block", cell="hex20", nx=25, ny=11, nz=11, nincs=1),
        # the benchmark's block: 2.0 M DOFs, lognormal stiffness, one linear increment
        dict(name="block_hex20_100x40x40", kind="block", cell="hex20", nx=100, ny=40, nz=40, nincs=1),
        # nonlinear geomechanics: the benchmark's von Mises slope on jittered TET10 cells, gravity and surcharge in
        # increments, the tangent assembled and the hierarchy built at every Newton iteration
        dict(name="slope_vm_tet10_24x5x10", kind="slope", cell="tet10", nx=24, ny=5, nz=10, nincs=5),
        # a parameter study: independent plane-strain models solved together, the persistent block-Jacobi launch
        dict(name="batch_quad8_64_mixed", kind="batch", cell="quad8", count=64, nmin=10, nmax=60, mix=1, solver="mixed"),
        # a larger study with the joined model's multigrid
        dict(name="batch_quad8_200_amg", kind="batch", cell="quad8", count=200, nmin=10, nmax=60, mix=2, solver="amg"),
        # mount_K as a plug-in of the reference: K assembled in the reference's operation order and handed over in its
        # CSC layout, on a jittered mesh
        dict(name="mount_hex8_29x13x13", kind="mount", cell="hex8", nx=29, ny=13, nz=13),
        # update_state!: internal forces and the von Mises return mapping for a given displacement, and the states
        # read back
        dict(name="update_vm_hex20_31x13x13", kind="update", cell="hex20", nx=31, ny=13, nz=13),
        # output: nodal patch recovery of all stress and strain fields
        dict(name="recover_hex20_41x17x17", kind="recover", cell="hex20", nx=41, ny=17, nz=17),
        # a Newmark stage of five increments with Rayleigh damping, multigrid solver
        dict(name="dynamic_hex20_21x9x9", kind="dynamic", cell="hex20", nx=21, ny=9, nz=9, nincs=5),
        # serving: a burst of requests of mixed sizes, 20 % of them elastoplastic, admitted as slots get free
        dict(name="serve_burst_10", kind="serve", cell="hex8", count=10, dofs_min=1000, dofs_max=60000, mix=3),
    ]


def _split(rng, cell, lo, hi):
    """Divisions of a block of lo..hi cells (log-uniform), longer in x, as the listed ones."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if cell.startswith("quad"):
        a = rng.uniform(1.0, 6.0)
        return dict(nx=max(3, round(math.sqrt(n * a))), ny=max(3, round(math.sqrt(n / a))))
    if cell == "tet10":  # six cells to a box
        n /= 6
    a = rng.uniform(1.0, 3.0)
    c = (n / a) ** (1.0 / 3.0)
    return dict(nx=max(3, round(a * c)), ny=max(3, round(c)), nz=max(3, round(c * rng.uniform(0.8, 1.25))))


def draw(rng):
    kind = rng.choice(["analysis", "beam", "block", "block", "slope", "batch", "batch", "mount", "update", "recover",
                       "dynamic", "serve"])
    if kind == "analysis":
        c = dict(cell="hex8", **_split(rng, "hex8", 60, 3000))
    elif kind == "beam":
        cell = rng.choice(["quad4", "quad8"])
        c = dict(cell=cell, nx=rng.randint(20, 120), ny=rng.randint(3, 12), nincs=rng.randint(5, 8))
    elif kind == "block":
        cell = rng.choice(["hex8", "hex20"])
        c = dict(cell=cell, nincs=rng.choice([1, 1, 2, 3]), **_split(rng, cell, 200, 30000))
    elif kind == "slope":
        k = rng.uniform(0.6, 1.3)
        c = dict(cell="tet10", nx=round(24 * k), ny=rng.randint(3, 6), nz=2 * round(5 * k), nincs=5)
    elif kind == "batch":
        solver = rng.choice(["mixed", "amg"])
        lo = rng.randint(4, 24)
        c = dict(cell="quad8", count=round(math.exp(rng.uniform(math.log(6), math.log(200)))), nmin=lo,
                 nmax=lo + rng.randint(4, 36), mix=rng.randint(10, 10 ** 6), solver=solver)
    elif kind == "mount":
        c = dict(cell="hex8", **_split(rng, "hex8", 100, 8000))
    elif kind == "update":
        cell = rng.choice(["hex8", "hex20", "tet10"])
        c = dict(cell=cell, **_split(rng, cell, 200, 6000))
    elif kind == "recover":
        cell = rng.choice(["hex8", "hex20"])
        c = dict(cell=cell, **_split(rng, cell, 100, 15000))
    elif kind == "dynamic":
        cell = rng.choice(["hex8", "hex20"])
        c = dict(cell=cell, nincs=rng.randint(3, 6), **_split(rng, cell, 100, 2500))
    else:
        c = dict(cell="hex8", count=rng.randint(4, 12), dofs_min=1000, dofs_max=round(math.exp(rng.uniform(math.log(8e3),
                                                                                                          math.log(6e4)))),
                 mix=rng.randint(10, 10 ** 6))
    return dict(kind=kind, **c)


# ---------------------------------------------------------------------------------------------------------------
# inputs: meshes, parameters and boundary conditions, from the case and the seed
# ---------------------------------------------------------------------------------------------------------------
_BOX = {"analysis": (1.0, 0.2, 0.2), "block": (10.0, 4.0, 4.0), "mount": (1.0, 0.4, 0.4), "update": (1.0, 0.4, 0.4),
        "recover": (10.0, 4.0, 4.0), "dynamic": (10.0, 4.0, 4.0)}


def _mesh3(case):
    b = _BOX[case["kind"]]
    return A.Mesh(A.Block([[0, 0, 0], list(b)], nx=case["nx"], ny=case["ny"], nz=case["nz"],
                          cellshape=_CELL[case["cell"]]))


def _conn(mesh):
    return np.concatenate(mesh.conn_list) if len(mesh.conn_list) > 1 else mesh.conn_list[0]


def _solid_inputs(case, seed):
    """A 3-D block: (mesh, E per cell, load q, fixed axis)."""
    rng = np.random.default_rng(seed)
    mesh = _mesh3(case)
    E = np.exp(rng.normal(math.log(30e3), 0.3, len(mesh.shape)))
    q = float(rng.uniform(0.5, 1.5))
    if case["kind"] == "mount":  # a distorted mesh: every entry of the element matrices is there
        c = np.array(mesh.coords)
        box = np.array(_BOX["mount"])
        h = (box / np.array([case["nx"], case["ny"], case["nz"]])).min()
        inside = ((c > 1e-9) & (c < box - 1e-9)).all(axis=1)
        c[inside] += rng.uniform(-0.15 * h, 0.15 * h, (int(inside.sum()), 3))
        mesh.coords = c
    return mesh, E, q, (0 if case["kind"] == "analysis" else 2)


def _block_bcs(case, q, axis):
    end = _BOX[case["kind"]][axis]
    a = "xyz"[axis]
    return [("%s==0" % a, A.SurfaceBC(ux=0, uy=0, uz=0)), ("%s==%r" % (a, end), A.SurfaceBC(tz=-q))]


def _batch_inputs(case, seed):
    """Rectangles 2 x 1 of n x n cells: the sizes belong to the case, E, nu and the load to the seed."""
    ns = np.random.default_rng(case["mix"]).integers(case["nmin"], case["nmax"] + 1, case["count"])
    rng = np.random.default_rng(seed)
    E = np.exp(rng.normal(math.log(200e3), 0.2, case["count"]))
    nu = rng.uniform(0.2, 0.35, case["count"])
    q = float(rng.uniform(0.5, 1.5))
    meshes = {}
    for n in ns:
        if int(n) not in meshes:
            meshes[int(n)] = A.Mesh(A.Block([[0, 0], [2.0, 1.0]], nx=int(n), ny=int(n), cellshape=L.QUAD8))
    return [int(n) for n in ns], meshes, E, nu, q


def _serve_inputs(case, seed):
    """Requests as in the serving benchmark: HEX8 blocks 1 x 0.5 x 0.5 in 1..4 increments, every fifth an
    elastoplastic TET10 block; sizes from the case, stiffness and load from the seed."""
    sizes = np.random.default_rng(case["mix"])
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["count"]):
        dofs = float(np.exp(sizes.uniform(np.log(case["dofs_min"]), np.log(case["dofs_max"]))))
        incs = int(sizes.integers(1, 5))
        s = float(np.exp(rng.normal(0.0, 0.2)))
        q = float(rng.uniform(0.5, 1.5))
        if i % 5 == 4:
            k = max(1, int(round(((min(dofs, 15e3) / 3) / 16) ** (1 / 3))))
            out.append(("tet10", 2 * k, k, incs, s, q))
        else:
            out.append(("hex8", 2 * max(1, int(round((dofs / 6) ** (1 / 3)))), max(1, int(round((dofs / 6) ** (1 / 3)))),
                        incs, s, q))
    return out


def _smooth(coords, rng, n):
    """n smooth seeded functions of the position: quadratics and a few waves."""
    x = coords / np.abs(coords).max()
    cols = [np.ones(len(x))] + [x[:, i] for i in range(3)] + [x[:, i] * x[:, j] for i in range(3) for j in range(i, 3)]
    cols += [np.sin(x @ rng.uniform(-4, 4, 3) + rng.uniform(0, 6)) for _ in range(4)]
    return np.stack(cols, 1) @ rng.normal(size=(len(cols), n))


# ---------------------------------------------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------------------------------------------
def _stage_params(case, **kw):
    return L.default_stage_params(nincs=case.get("nincs", 1),
                                  linear=L.default_solve_opts(method=_METHOD[case.get("solver", "amg")], rtol=RTOL), **kw)


def prepare(case, seed):
    kind, s = case["kind"], dict(case=case)
    rng = np.random.default_rng(seed)
    if kind in ("analysis", "block", "mount", "dynamic"):
        mesh, E, q, axis = _solid_inputs(case, seed)
        s["bcs"] = _block_bcs(case, q, axis)
        s["model"] = model = A.FEModel(mesh, [("all", A.LinearElastic(E=30e3, nu=0.2, rho=2.4e-3))],
                                       nips=_NIP[case["cell"]], E=E)
        if kind in ("block", "mount"):
            setup = model.configure_dofs(s["bcs"])
            if kind == "block":
                s["Uex"], s["Fex"] = model.get_bc_vals(setup)
                s["params"] = _stage_params(case)
    elif kind == "beam":
        mesh = A.Mesh(A.Block([[0, 0], [1.0, 0.1]], nx=case["nx"], ny=case["ny"], cellshape=_CELL[case["cell"]]))
        ne = len(mesh.shape)
        s["model"] = model = A.FEModel(mesh, [("all", A.VonMises(E=210e6, nu=0.3, fy=240e3, H=30e6))],
                                       A.MechContext(stressmodel="planestress"), thickness=0.05,
                                       nips=_NIP[case["cell"]], E=210e6 * np.exp(rng.normal(0.0, 0.05, ne)))
        setup = model.configure_dofs([("x==0", A.NodeBC(ux=0, uy=0)),
                                      ("x==1", A.NodeBC(uy=float(rng.uniform(-0.0097, -0.0093))))])
        s["Uex"], s["Fex"] = model.get_bc_vals(setup)
        s["state0"] = model.state()
        s["params"] = _stage_params(dict(case, solver="mixed"), maxits=20)
    elif kind == "slope":
        g, n = workloads.SLOPE, (case["nx"], case["ny"], case["nz"])
        mesh = A.Mesh(A.Block([[0, 0, 0], [g["L"], g["W"], g["H"]]], nx=n[0], ny=n[1], nz=n[2], cellshape=L.TET10))
        mesh.coords = workloads.slope_coords(mesh.coords, mesh.elem_nodes(), workloads.boundary_nodes(mesh), 4, *n,
                                             seed=seed)
        s["model"] = model = A.FEModel(mesh, [("all", A.VonMises(E=50e3, nu=0.3, fy=100.0, H=1e3))])
        setup = model.configure_dofs(workloads.slope_bcs(A, float(rng.uniform(110.0, 130.0))))
        s["Uex"], s["Fex"] = model.get_bc_vals(setup)
        s["state0"] = model.state()
        s["params"] = _stage_params(case, tol=1e-6, maxits=20)
    elif kind == "batch":
        ns, meshes, E, nu, q = _batch_inputs(case, seed)
        ctx = A.MechContext(stressmodel="planestrain")
        models = [A.FEModel(meshes[n], [("all", A.LinearElastic(E=float(e), nu=float(v)))], ctx, nips=9, device=False)
                  for n, e, v in zip(ns, E, nu)]
        s["batch"] = ba = A.BatchAnalysis(models)
        ba.addstage([("x==0", A.SurfaceBC(ux=0, uy=0)), ("x==2", A.SurfaceBC(tx=q))])
        s["Uex"], s["Fex"] = ba.configure(ba.stages[0].bcs)
        s["model"], s["params"] = ba.joined, _stage_params(case)
    elif kind == "update":
        mesh = _mesh3(case)
        E = np.exp(rng.normal(math.log(200e3), 0.1, len(mesh.shape)))
        s["model"] = model = A.FEModel(mesh, [("all", A.VonMises(E=200e3, nu=0.3, fy=200.0, H=2e3))],
                                       nips=_NIP[case["cell"]], E=E)
        model.configure_dofs([("x==0", A.SurfaceBC(ux=0, uy=0, uz=0))])
        u = 4e-4 * _smooth(mesh.coords, rng, 3)
        s["dU"] = u[model.dof_node, model.dof_comp]
    elif kind == "recover":
        mesh = _mesh3(case)
        s["model"] = model = A.FEModel(mesh, [("all", A.LinearElastic(E=30e3, nu=0.2))], nips=_NIP[case["cell"]])
        model.configure_dofs([("z==0", A.SurfaceBC(ux=0, uy=0, uz=0))])
        model.set_state(_recover_state(case, mesh, seed))
    elif kind == "serve":
        s["server"] = serve.Server(hbm_budget_bytes=60e9, max_active=8)
        s["requests"] = []
        for cell, nx, k, incs, sc, q in _serve_inputs(case, seed):
            mesh = A.Mesh(A.Block([[0, 0, 0], [1.0, 0.5, 0.5]], nx=nx, ny=k, nz=k, cellshape=_CELL[cell]))
            kw = dict(nincs=incs, solver="amg", linear_rtol=RTOL)
            if cell == "tet10":
                m = A.FEModel(mesh, [("all", A.VonMises(E=50e3 * sc, nu=0.3, fy=100.0, H=1e3))], device=False)
                bcs = [("z==0", A.SurfaceBC(ux=0, uy=0, uz=0)), ("z==0.5", A.SurfaceBC(tz=-80.0 - 10.0 * q)),
                       ("all", A.BodyC(wz=-20.0))]
            else:
                m = A.FEModel(mesh, [("all", A.LinearElastic(E=200e3 * sc, nu=0.3))], device=False)
                bcs = [("x==0", A.SurfaceBC(ux=0, uy=0, uz=0)), ("x==1", A.SurfaceBC(tz=-q))]
            s["requests"].append((m, bcs, kw))
    else:
        raise ValueError(kind)
    return s


def run(s):
    kind = s["case"]["kind"]
    model = s.get("model")
    if kind in ("block", "batch"):
        rc, U, F, _ = model.dev.stage_run(s["Uex"], s["Fex"], s["params"])
        if rc:
            raise RuntimeError(model.dev.last_error())
        return [U, F]
    if kind in ("beam", "slope"):  # the stage starts from the given states
        model.set_state(s["state0"])
        rc, U, F, _ = model.dev.stage_run(s["Uex"], s["Fex"], s["params"])
        if rc:
            raise RuntimeError(model.dev.last_error())
        return [U, F, model.state()]
    if kind == "analysis":
        ana = A.MechAnalysis(model)
        ana.addstage(s["bcs"])
        ok, msg = ana.solve(linear_rtol=RTOL)
        if not ok:
            raise RuntimeError(msg)
        return [model.U, model.F]
    if kind == "mount":
        K = model.mount_K()
        return [K.indptr, K.indices, K.data]
    if kind == "update":
        return [model.update_state(s["dU"]), model.state()]
    if kind == "recover":
        V, _ = model.nodal_patch_recovery()
        return V
    if kind == "dynamic":
        ana = A.DynAnalysis(model)
        ana.addstage(s["bcs"], nincs=s["case"]["nincs"], tspan=0.002 * s["case"]["nincs"])
        ok, msg = ana.solve(solver="amg", linear_rtol=RTOL, alpha=0.5, beta=1e-4)
        if not ok:
            raise RuntimeError(msg)
        return [model.U, model.V, model.A, model.F]
    tickets = [s["server"].submit(m, bcs, **kw) for m, bcs, kw in s["requests"]]
    out = []
    for t in tickets:
        rc, U, F, _, msg = s["server"].wait(t)
        if rc:
            raise RuntimeError(msg)
        out.append([U, F])
    return out


# ---------------------------------------------------------------------------------------------------------------
# work: inputs read once, outputs written once, and the arithmetic of one element integration
# ---------------------------------------------------------------------------------------------------------------
def _counts(cell, nx, ny, nz=0):
    """(cells, nodes) of a structured block."""
    if cell == "quad4":
        return nx * ny, (nx + 1) * (ny + 1)
    if cell == "quad8":
        return nx * ny, (nx + 1) * (ny + 1) + nx * (ny + 1) + (nx + 1) * ny
    if cell == "hex8":
        return nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)
    if cell == "tet10":
        return 6 * nx * ny * nz, (2 * nx + 1) * (2 * ny + 1) * (2 * nz + 1)
    v = (nx + 1) * (ny + 1) * (nz + 1)
    return nx * ny * nz, v + nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz


def _solid_work(kind, cell, ne, nn, passes):
    d = 2 if cell.startswith("quad") else 3
    nen, nip = _NEN[cell], _NIP[cell]
    mesh = nn * d * 8 + ne * nen * 4 + ne * 8
    vec = nn * d * 8
    stiff = ne * nip * nen * (nen + 1) / 2 * 2 * d * d  # pairs a <= b of w g_a g_b'
    internal = ne * nip * nen * 2 * (2 * d * d)         # strains and B' sigma
    state = ne * nip * 16 * 8
    if kind == "mount":
        return mesh + nn * d * 27 * d * 16, stiff
    if kind == "update":
        return mesh + 2 * vec + state, internal
    if kind == "recover":
        return mesh + ne * nip * 12 * 8 + nn * 16 * 8, 2.0 * ne * nip * 8 * 16 * 7
    if kind == "dynamic":
        return mesh + 6 * vec, 2 * stiff + passes * internal
    if kind in ("beam", "slope"):
        return mesh + 4 * vec + 2 * state, passes * (stiff + internal)
    return mesh + 4 * vec, stiff + passes * internal


def work(case):
    kind, cell = case["kind"], case["cell"]
    b = f = 0.0
    if kind == "batch":
        for n in np.random.default_rng(case["mix"]).integers(case["nmin"], case["nmax"] + 1, case["count"]):
            w = _solid_work(kind, cell, *_counts(cell, int(n), int(n)), 1)
            b, f = b + w[0], f + w[1]
    elif kind == "serve":
        for c, nx, k, incs, _, _ in _serve_inputs(case, 0):
            w = _solid_work("slope" if c == "tet10" else kind, c, *_counts(c, nx, k, k), incs)
            b, f = b + w[0], f + w[1]
    else:
        b, f = _solid_work(kind, cell, *_counts(cell, case["nx"], case["ny"], case.get("nz", 0)), case.get("nincs", 1))
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------------------------------------------------------
# exact: the same problems in 64 bits
# ---------------------------------------------------------------------------------------------------------------
_CORNERS = {2: [[-1, -1], [1, -1], [1, 1], [-1, 1]],
            3: [[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]]}
_EDGES = {"quad8": [(0, 1), (1, 2), (2, 3), (3, 0)],
          "hex20": [(0, 1), (1, 2), (2, 3), (3, 0), (4, 5), (5, 6), (6, 7), (7, 4), (0, 4), (1, 5), (2, 6), (3, 7)],
          "tet10": [(0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3)]}


def _monomials(cell):
    """Exponents of the monomials that span the cell's shape functions."""
    if cell == "tet10":
        return [(i, j, k) for i in range(3) for j in range(3) for k in range(3) if i + j + k <= 2]
    d = 2 if cell.startswith("quad") else 3
    full = [e for e in np.ndindex(*([3] * d))]
    if cell in ("quad4", "hex8"):
        return [e for e in full if max(e) <= 1]
    return [e for e in full if sum(1 for v in e if v == 2) <= 1]  # serendipity: one square at most


def _shape_tables(cell):
    """(N (nip, nen), dN/dR (nip, nen, d), w (nip)) in 64 bits, from the cell's node positions."""
    if cell == "tet10":
        v = [[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]]
        d = 3
    else:
        d = 2 if cell.startswith("quad") else 3
        v = _CORNERS[d]
    P = [list(map(float, p)) for p in v]
    P += [[(P[a][i] + P[b][i]) / 2 for i in range(d)] for a, b in _EDGES.get(cell, [])]
    P = np.array(P)
    ex = _monomials(cell)

    def mono(X):
        return np.stack([np.prod([X[:, i] ** e[i] for i in range(d)], axis=0) for e in ex], 1)

    def dmono(X, k):
        return np.stack([np.prod([(X[:, i] ** e[i] if i != k else (e[i] * X[:, i] ** max(e[i] - 1, 0))) for i in range(d)],
                                 axis=0) for e in ex], 1)
    C = np.linalg.inv(mono(P))
    if cell == "tet10":
        s5 = math.sqrt(5.0)
        a, b = (5 + 3 * s5) / 20, (5 - s5) / 20
        R, w = np.array([[a, b, b], [b, a, b], [b, b, a], [b, b, b]]), np.full(4, 1 / 24)
    else:
        pts, ws = np.polynomial.legendre.leggauss({4: 2, 9: 3, 8: 2, 27: 3}[_NIP[cell]])
        grid = np.meshgrid(*([np.arange(len(pts))] * d), indexing="ij")
        idx = np.stack([g.ravel() for g in grid[::-1]], 1)  # the first coordinate fastest
        R, w = pts[idx], np.prod(ws[idx], axis=1)
    return mono(R) @ C, np.stack([dmono(R, k) @ C for k in range(d)], 2), w


_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=_DEV)


class _Fem:
    """Linear elastic solids in 64 bits: element matrices and their sum applied to a vector."""

    def __init__(self, cell, coords, conn, E, nu):
        self.d = d = 2 if cell.startswith("quad") else 3
        self.nn, self.ne = len(coords), len(conn)
        N, D, w = _shape_tables(cell)
        self.N = _t(N)
        self.conn = _t(conn, torch.int64)
        self.dof = (self.conn[:, :, None] * d + torch.arange(d, device=_DEV)).reshape(self.ne, -1)
        X, self.E = _t(coords[:, :d]), _t(np.broadcast_to(E, self.ne))
        self.nu = _t(np.broadcast_to(nu, self.ne))
        J = torch.einsum("eai,qaj->eqij", X[self.conn], _t(D))
        self.w = torch.linalg.det(J) * _t(w)
        self.g = torch.einsum("qaj,eqji->eqai", _t(D), torch.linalg.inv(J))

    def strain(self, u):
        """Mandel strains (ne, nip, 6) of node displacements u (nn, 3)."""
        G = torch.einsum("eqai,eaj->eqij", self.g, u[self.conn])
        e = 0.5 * (G + G.transpose(2, 3))
        r = math.sqrt(2.0)
        return torch.stack([e[..., 0, 0], e[..., 1, 1], e[..., 2, 2], r * e[..., 1, 2], r * e[..., 0, 2], r * e[..., 0, 1]], -1)

    def stiffness(self):
        lam = self.E * self.nu / ((1 + self.nu) * (1 - 2 * self.nu))
        mu = self.E / (2 * (1 + self.nu))
        eye = torch.eye(self.d, dtype=torch.float64, device=_DEV)
        out = []
        for s in range(0, self.ne, 20000):
            g, w = self.g[s:s + 20000], self.w[s:s + 20000]
            T = torch.einsum("eq,eqai,eqbj->eaibj", w, g, g)
            la, m = lam[s:s + 20000, None, None, None, None], mu[s:s + 20000, None, None, None, None]
            K = la * T + m * T.permute(0, 1, 4, 3, 2)
            K += m * torch.einsum("eakbk,ij->eaibj", T, eye)
            out.append(K.reshape(len(g), self.dof.shape[1], -1))
        return torch.cat(out)

    def mass(self, rho):
        m = torch.einsum("eq,qa,qb->eab", self.w * rho, self.N, self.N)
        eye = torch.eye(self.d, dtype=torch.float64, device=_DEV)
        return torch.einsum("eab,ij->eaibj", m, eye).reshape(self.ne, self.dof.shape[1], -1)

    def mul(self, Ke, u):
        f = torch.bmm(Ke, u[self.dof].unsqueeze(2)).reshape(-1)
        return torch.zeros_like(u).index_add_(0, self.dof.reshape(-1), f)

    def solve(self, Ke, b, free):
        """x with (sum Ke x) = b at free DOFs and 0 elsewhere: conjugate gradients, diagonal preconditioner."""
        dg = torch.zeros_like(b).index_add_(0, self.dof.reshape(-1),
                                            torch.diagonal(Ke, dim1=1, dim2=2).reshape(-1))
        inv = torch.where(free, 1.0 / dg, torch.zeros_like(dg))
        r = torch.where(free, b, torch.zeros_like(b))
        x, z = torch.zeros_like(b), inv * r
        p, rz, b2 = z.clone(), torch.dot(r, z), float(torch.dot(r, r))
        for it in range(1, 30001):
            q = torch.where(free, self.mul(Ke, p), torch.zeros_like(b))
            a = rz / torch.dot(p, q)
            x += a * p
            r -= a * q
            if it % 50 == 0 and float(torch.dot(r, r)) <= 1e-28 * b2:
                break
            z = inv * r
            rz, old = torch.dot(r, z), rz
            p = z + (rz / old) * p
        return x


_SIDE = {"quad4": (2, 1, [(0,), (1,)]), "quad8": (3, 1, [(0,), (1,), (2,)]),
         "hex8": (4, 2, [(0, 0), (1, 0), (0, 1), (1, 1)]),
         "hex20": (8, 2, [(0, 0), (1, 0), (0, 1), (1, 1), (2, 0), (0, 2), (2, 1), (1, 2)])}


def _face_load(cell, mesh, axis, value, comp, q):
    """Nodal forces of a uniform traction q in direction comp on the side coord[axis] == value, by Gauss rules of two
    points a direction, the rule of the reference's facets."""
    d = mesh.ndim
    npt, fd, ex = _SIDE[cell]
    table = (mesh.edge_nodes if d == 2 else mesh.face_nodes)[:, :npt]
    tb = table[(np.abs(mesh.coords[table][:, :, axis] - value) < 1e-9).all(axis=1)]
    if fd == 1:
        P = np.array([[-1.0], [1.0], [0.0]])[:npt]
    else:
        P = np.array([[-1, -1], [1, -1], [1, 1], [-1, 1], [0, -1], [1, 0], [0, 1], [-1, 0]], dtype=float)[:npt]
    g = 1 / math.sqrt(3.0)
    R = np.array([[a] for a in (-g, g)] if fd == 1 else [[a, b] for b in (-g, g) for a in (-g, g)])

    def mono(X, k=None):
        return np.stack([np.prod([X[:, i] ** e[i] if i != k else e[i] * X[:, i] ** max(e[i] - 1, 0)
                                  for i in range(fd)], axis=0) for e in ex], 1)
    C = np.linalg.inv(mono(P))
    T = [np.einsum("qa,fai->fqi", mono(R, k) @ C, mesh.coords[tb]) for k in range(fd)]
    size = np.linalg.norm(T[0] if fd == 1 else np.cross(T[0], T[1]), axis=2)
    F = np.zeros((len(mesh.coords), d))
    np.add.at(F[:, comp], tb.reshape(-1), (q * np.einsum("fq,qa->fa", size, mono(R) @ C)).reshape(-1))
    return F


def _in_order(v, presc):
    """A (nn, d) array in the order of the DOF numbering: unknowns first, node by node, then prescribed ones."""
    p = presc.reshape(-1)
    return v.reshape(-1)[np.concatenate([np.nonzero(~p)[0], np.nonzero(p)[0]])]


def _linear(cell, mesh, conn, E, nu, presc, F):
    """U and the forces K U, (nn, d), of a linear stage."""
    fem = _Fem(cell, mesh.coords, conn, E, nu)
    Ke = fem.stiffness()
    x = fem.solve(Ke, _t(F).reshape(-1), _t(~presc, torch.bool).reshape(-1))
    return x.cpu().numpy().reshape(F.shape), fem.mul(Ke, x).cpu().numpy().reshape(F.shape)


def exact(case, seed):
    kind, cell = case["kind"], case["cell"]
    if kind in ("beam", "slope"):
        return None
    if kind in ("analysis", "block"):
        mesh, E, q, axis = _solid_inputs(case, seed)
        presc = np.repeat((np.abs(mesh.coords[:, axis]) < 1e-9)[:, None], 3, 1)
        F = _face_load(cell, mesh, axis, _BOX[kind][axis], 2, -q)
        U, R = _linear(cell, mesh, _conn(mesh), E, 0.2, presc, F)
        return [U, R] if kind == "analysis" else [_in_order(U, presc), _in_order(R, presc)]
    if kind == "batch":
        ns, meshes, E, nu, q = _batch_inputs(case, seed)
        joined = A.Mesh.join([meshes[n] for n in ns])[0]
        per = np.array([len(meshes[n].shape) for n in ns])
        presc = np.repeat((np.abs(joined.coords[:, 0]) < 1e-9)[:, None], 2, 1)
        F = _face_load(cell, joined, 0, 2.0, 0, q)
        U, R = _linear(cell, joined, _conn(joined), np.repeat(E, per), np.repeat(nu, per), presc, F)
        return [_in_order(U, presc), _in_order(R, presc)]
    if kind == "serve":
        out = []
        for c, nx, k, incs, sc, q in _serve_inputs(case, seed):
            if c == "tet10":
                out.append([None, None])
                continue
            mesh = A.Mesh(A.Block([[0, 0, 0], [1.0, 0.5, 0.5]], nx=nx, ny=k, nz=k, cellshape=_CELL[c]))
            presc = np.repeat((np.abs(mesh.coords[:, 0]) < 1e-9)[:, None], 3, 1)
            out.append(list(_linear(c, mesh, _conn(mesh), 200e3 * sc, 0.3, presc, _face_load(c, mesh, 0, 1.0, 2, -q))))
        return out
    if kind == "mount":
        mesh, E, _, axis = _solid_inputs(case, seed)
        fem = _Fem(cell, mesh.coords, _conn(mesh), E, 0.2)
        presc = np.repeat((np.abs(mesh.coords[:, axis]) < 1e-9)[:, None], 3, 1)
        n = presc.size
        eq = torch.empty(n, dtype=torch.int64, device=_DEV)
        eq[_t(_in_order(np.arange(n), presc), torch.int64)] = torch.arange(n, device=_DEV)
        e = eq[fem.dof]
        key = (e[:, None, :] * n + e[:, :, None]).reshape(-1)  # column-major
        u, inv = torch.unique(key, return_inverse=True)
        val = torch.zeros(len(u), dtype=torch.float64, device=_DEV).index_add_(0, inv, fem.stiffness().reshape(-1))
        return [None, None, val.cpu().numpy()]
    if kind == "update":
        return _exact_update(case, seed)
    if kind == "recover":
        return _exact_recover(case, seed)
    return _exact_dynamic(case, seed)


def _exact_update(case, seed):
    """Internal forces and states of the von Mises update from zero states."""
    rng = np.random.default_rng(seed)
    mesh = _mesh3(case)
    E = np.exp(rng.normal(math.log(200e3), 0.1, len(mesh.shape)))
    u = 4e-4 * _smooth(mesh.coords, rng, 3)
    fem = _Fem(case["cell"], mesh.coords, _conn(mesh), E, 0.3)
    fy, H, nu = 200.0, 2e3, 0.3
    eps = fem.strain(_t(u))
    E_ = fem.E[:, None]
    mu, K = E_ / (2 * (1 + nu)), E_ / (3 * (1 - 2 * nu))
    p = eps[..., :3].sum(-1)
    one = torch.tensor([1.0, 1, 1, 0, 0, 0], dtype=torch.float64, device=_DEV)
    s = 2 * mu[..., None] * (eps - p[..., None] / 3 * one)
    ns = torch.linalg.vector_norm(s, dim=-1)
    f = math.sqrt(1.5) * ns - fy
    dl = torch.where(f < 1e-8, torch.zeros_like(f), f / (3 * mu + math.sqrt(1.5) * H))
    s = s * (1 - math.sqrt(6.0) * mu * dl / ns)[..., None]
    sig = (K * p)[..., None] * one + s
    r = math.sqrt(2.0)
    t = torch.stack([sig[..., 0], sig[..., 5] / r, sig[..., 4] / r, sig[..., 5] / r, sig[..., 1], sig[..., 3] / r,
                     sig[..., 4] / r, sig[..., 3] / r, sig[..., 2]], -1).reshape(*sig.shape[:2], 3, 3)
    fe = torch.einsum("eq,eqai,eqij->eaj", fem.w, fem.g, t).reshape(-1)
    F = torch.zeros(3 * fem.nn, dtype=torch.float64, device=_DEV).index_add_(0, fem.dof.reshape(-1), fe)
    presc = np.repeat((np.abs(mesh.coords[:, 0]) < 1e-9)[:, None], 3, 1)
    z = torch.zeros_like(dl)[..., None]
    st = torch.cat([sig, eps, dl[..., None], dl[..., None], z, z], -1).reshape(-1, 16)
    return [_in_order(F.cpu().numpy().reshape(-1, 3), presc), st.cpu().numpy()]


def _recover_state(case, mesh, seed):
    """Stresses and strains at the integration points: smooth fields and a little noise."""
    rng = np.random.default_rng(seed)
    N, _, _ = _shape_tables(case["cell"])
    ip = np.einsum("qa,eai->eqi", N, mesh.coords[_conn(mesh)]).reshape(-1, 3)
    st = np.zeros((len(ip), 16))
    st[:, :6] = 10.0 * _smooth(ip, rng, 6) + 0.1 * rng.normal(size=(len(ip), 6))
    st[:, 6:12] = 1e-3 * _smooth(ip, rng, 6) + 1e-5 * rng.normal(size=(len(ip), 6))
    return st


def _exact_recover(case, seed):
    """A fit of 1, x, y, z, xy, yz, xz over the eight cells of every inner corner node, averaged over the patches that
    reach a node (with two or more cells a side, inner patches reach every node)."""
    mesh = _mesh3(case)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    conn, coords = _t(_conn(mesh), torch.int64), _t(mesh.coords)
    N, _, _ = _shape_tables(case["cell"])
    nip = len(N)
    st = _t(_recover_state(case, mesh, seed))
    r = math.sqrt(2.0)
    sg, ep = st[:, :6].clone(), st[:, 6:12].clone()
    sg[:, 3:] /= r
    ep[:, 3:] /= r
    T = torch.stack([sg[:, 0], sg[:, 5], sg[:, 4], sg[:, 5], sg[:, 1], sg[:, 3], sg[:, 4], sg[:, 3], sg[:, 2]], 1)
    ev = _eig3(T.reshape(-1, 3, 3))
    mises = torch.sqrt(0.5 * ((sg[:, 0] - sg[:, 1]) ** 2 + (sg[:, 1] - sg[:, 2]) ** 2 + (sg[:, 2] - sg[:, 0]) ** 2)
                       + 3 * (sg[:, 3:] ** 2).sum(1))
    W = torch.cat([sg, mises[:, None], ev, ep], 1).reshape(len(conn), nip, 16)
    ip = torch.einsum("qa,eai->eqi", _t(N), coords[conn])
    # the cell at (i, j, k) is number i + nx (j + ny k)
    i, j, k = np.meshgrid(np.arange(nx - 1), np.arange(ny - 1), np.arange(nz - 1), indexing="ij")
    first = (i + nx * (j + ny * k)).ravel()
    cells = first[:, None] + np.array([a + nx * (b + ny * c) for a in (0, 1) for b in (0, 1) for c in (0, 1)])
    cells = _t(cells, torch.int64)
    V = torch.zeros(len(coords), 16, dtype=torch.float64, device=_DEV)
    cnt = torch.zeros(len(coords), dtype=torch.float64, device=_DEV)

    def basis(x):
        return torch.stack([torch.ones_like(x[..., 0]), x[..., 0], x[..., 1], x[..., 2], x[..., 0] * x[..., 1],
                            x[..., 1] * x[..., 2], x[..., 0] * x[..., 2]], -1)
    for s in range(0, len(cells), 2000):
        c = cells[s:s + 2000]
        x = ip[c].reshape(len(c), -1, 3)
        mid, sc = x.mean(1, keepdim=True), (x.amax(1, keepdim=True) - x.amin(1, keepdim=True)) / 2
        Q, R = torch.linalg.qr(basis((x - mid) / sc))
        co = torch.linalg.solve_triangular(R, Q.transpose(1, 2) @ W[c].reshape(len(c), -1, 16), upper=True)
        nodes = conn[c].reshape(len(c), -1)
        srt, order = torch.sort(nodes, 1)
        once = torch.ones_like(srt, dtype=torch.bool)
        once[:, 1:] = srt[:, 1:] != srt[:, :-1]
        val = basis((coords[srt] - mid) / sc) @ co
        V.index_add_(0, srt[once], val[once])
        cnt.index_add_(0, srt[once], torch.ones_like(srt[once], dtype=torch.float64))
    return (V / cnt[:, None]).cpu().numpy()


def _eig3(T):
    """Eigenvalues of symmetric 3 x 3 matrices, largest first."""
    return torch.cat([torch.linalg.eigvalsh(t) for t in torch.split(T, 50000)]).flip(1)


def _exact_dynamic(case, seed):
    """Newmark's average acceleration with C = 0.5 M + 1e-4 K from rest under a constant load."""
    mesh, E, q, axis = _solid_inputs(case, seed)
    fem = _Fem(case["cell"], mesh.coords, _conn(mesh), E, 0.2)
    free = torch.ones(fem.nn, 3, dtype=torch.bool, device=_DEV)
    free[_t(np.abs(mesh.coords[:, axis]) < 1e-9, torch.bool)] = False
    free = free.reshape(-1)
    F = _t(_face_load(case["cell"], mesh, axis, _BOX["dynamic"][axis], 2, -q)).reshape(-1)
    Ke, Me = fem.stiffness(), fem.mass(2.4e-3)
    Ce = 0.5 * Me + 1e-4 * Ke
    dt = 0.002
    Kp = Ke + 4 / dt ** 2 * Me + 2 / dt * Ce
    U, V = torch.zeros_like(F), torch.zeros_like(F)
    a = fem.solve(Me, F, free)
    for _ in range(case["nincs"]):
        b = F + fem.mul(Me, 4 / dt ** 2 * U + 4 / dt * V + a) + fem.mul(Ce, 2 / dt * U + V)
        Un = fem.solve(Kp, b, free)
        a = torch.where(free, 4 / dt ** 2 * (Un - U) - 4 / dt * V - a, torch.zeros_like(a))
        V = torch.where(free, 2 / dt * (Un - U) - V, torch.zeros_like(V))
        U = Un
    R = fem.mul(Ke, U) + fem.mul(Ce, V) + fem.mul(Me, a)
    return [v.cpu().numpy().reshape(-1, 3) for v in (U, V, a, R)]
