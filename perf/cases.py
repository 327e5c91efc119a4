"""The workloads that a user of this framework runs, as measurable cases.

Each case is one pass of a user's program through the public entry points (the
Python mirror of Elfel.jl's API, or the C ABI of include/elfel_gpu.h the way a
Julia binding calls it, with page-locked host buffers):

  reassemble    a resident system is assembled again with new coefficients and
                its K values and F come back to the host (a nonlinear or
                time-dependent driver whose solver lives on the host)
  assemble_csc  the reference's assembleKF + finish!: host mesh and DOF tables
                in, SparseMatrixCSC arrays and F out
  coo           the generic path for any weak form: triplets in, CSC out
  script        a whole driver script (test/test_heat.jl): set-up, assembly and
                solve! of a small problem, T out
  solve         a resident system re-assembled with new coefficients and solved
                on the device (solve!), T out
  serve         a closed-loop burst of heat requests through the server

Meshes are the block meshes of the reference's tests (interior vertices moved
by a seeded +-0.2h, conductivity log-uniform in [0.5, 2], T = 1 + x^2 + 2 y^2
on the boundary), the plane-strain cantilever and the lid-driven Taylor-Hood
cavity.  Solves run to a relative residual of 1e-12, which keeps the solution
error well below 1e-8.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import __graft_entry__  # noqa: E402

E = __graft_entry__.package()
N = E._native

Q = -6.0
RTOL = 1e-12


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a teaching-size script, every call new: latency and launches
        {"name": "script T3 12", "kind": "script", "problem": "T3", "n": 12, "method": "pcg64"},
        # the smallest resident re-assembly: latency
        {"name": "reassemble T6 24", "kind": "reassemble", "problem": "T6", "n": 24},
        # the benchmark's 2M-element heat system, assembled again and again
        {"name": "reassemble T6 1000", "kind": "reassemble", "problem": "T6", "n": 1000},
        # two unknowns per node: load stepping on the cantilever
        {"name": "reassemble elasticity 500", "kind": "reassemble", "problem": "elasticity", "n": 500},
        # the Taylor-Hood cavity's three blocks
        {"name": "reassemble stokes 230", "kind": "reassemble", "problem": "stokes", "n": 230},
        # bilinear quadrilaterals, an odd size
        {"name": "reassemble Q4 701", "kind": "reassemble", "problem": "Q4", "n": 701},
        # the drop-in call: tables in, SparseMatrixCSC out, nothing resident before
        {"name": "assemble_csc T6 500", "kind": "assemble_csc", "problem": "T6", "n": 500},
        # a user's own weak form: 3.7M triplets through sparse()
        {"name": "coo T6 227", "kind": "coo", "problem": "T6", "n": 227},
        # one time step of a mid-size problem in FP64
        {"name": "solve T6 fp64 180", "kind": "solve", "problem": "T6", "n": 180, "method": "pcg64"},
        # a large solve with the default method
        {"name": "solve T6 fp32 ir 450", "kind": "solve", "problem": "T6", "n": 450, "method": "pcg32_ir"},
        # saddle-point solve
        {"name": "solve stokes 32", "kind": "solve", "problem": "stokes", "n": 32, "method": "minres64"},
        # serving: a burst of mixed requests, systems resident after the first
        {"name": "serve 32 to 96", "kind": "serve", "count": 32, "n": 96, "mix": 5},
    ]


#: Sizes that draw() covers, by kind and problem: cells per side.
RANGES = {
    ("script", "T3"): (4, 64), ("script", "T6"): (3, 40), ("script", "Q4"): (4, 64), ("script", "T4"): (3, 12),
    ("reassemble", "T3"): (12, 1000), ("reassemble", "T6"): (8, 1000), ("reassemble", "Q4"): (12, 1000),
    ("reassemble", "T4"): (4, 50), ("reassemble", "elasticity"): (8, 500), ("reassemble", "stokes"): (6, 230),
    ("assemble_csc", "T3"): (12, 700), ("assemble_csc", "T6"): (8, 500), ("assemble_csc", "Q4"): (12, 700),
    ("assemble_csc", "T4"): (4, 40), ("assemble_csc", "elasticity"): (8, 250), ("assemble_csc", "stokes"): (6, 140),
    ("coo", "T6"): (8, 227), ("coo", "T3"): (12, 400),
    ("solve", "T3"): (16, 500), ("solve", "T6"): (16, 300), ("solve", "Q4"): (16, 500), ("solve", "T4"): (6, 40),
    ("solve", "elasticity"): (8, 48), ("solve", "stokes"): (6, 32),
}


def draw(rng):
    kind = rng.choice(["script", "reassemble", "reassemble", "assemble_csc", "coo", "solve", "solve", "serve"])
    if kind == "serve":
        return {"kind": kind, "count": rng.randint(8, 32), "n": rng.randint(40, 96), "mix": rng.randrange(1 << 20)}
    problem = rng.choice([p for k, p in RANGES if k == kind])
    lo, hi = RANGES[kind, problem]
    c = {"kind": kind, "problem": problem, "n": int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))}
    if kind in ("script", "solve"):
        c["method"] = "minres64" if problem == "stokes" else rng.choice(["pcg64", "pcg32_ir"])
        if problem == "elasticity":
            c["method"] = "pcg64"
    return c


# ------------------------------------------------------------------ problems
def _tempf(xy):
    return 1.0 + xy[:, 0] ** 2 + 2.0 * xy[:, 1] ** 2


def _on_boundary(xy):
    """Mask of the nodes on the faces of the mesh's bounding box."""
    return ((xy == xy.min(axis=0)) | (xy == xy.max(axis=0))).any(axis=1)


class Problem:
    """Mesh, numbered spaces and tables of one (problem, n); coordinates before the jitter."""

    def __init__(self, problem, n):
        self.problem = problem
        self.pfesp = None
        if problem in ("T3", "T6", "Q4", "T4"):
            block = {"T3": E.T3block, "T6": E.T6block, "Q4": E.Q4block}.get(problem)
            mesh = E.T4block(1.0, 1.0, 1.0, n, n, n) if problem == "T4" else block(1.0, 1.0, n, n)
            fe = {"T3": E.FEH1_T3, "T6": E.FEH1_T6, "Q4": E.FEH1_Q4, "T4": E.FEH1_T4}[problem]()
            self.fesp = E.FESpace(float, mesh, fe)
            self.fixed = _on_boundary(mesh.xy)
            bn = np.nonzero(self.fixed)[0] + 1
            E.setebc(self.fesp, 0, bn, 1, _tempf(mesh.xy[bn - 1]))
            E.numberdofs(self.fesp)
            self.h = 1.0 / n
            self.rule = {"kind": "Gauss", "order": 2} if problem == "Q4" else {"npts": 1 if problem == "T4" else 3}
            spaces = self.fesp
        elif problem == "elasticity":  # n x n/2 cells of [0,2] x [0,1], left edge clamped
            m = max(1, n // 2)
            mesh = E.T6block(2.0, 1.0, n, m)
            self.fesp = E.FESpace(float, mesh, E.FEH1_T6(), 2)
            self.fixed = _on_boundary(mesh.xy)
            left = np.nonzero(mesh.xy[:, 0] == 0.0)[0] + 1
            E.setebc(self.fesp, 0, left, 1, 0.0)
            E.setebc(self.fesp, 0, left, 2, 0.0)
            E.numberdofs(self.fesp)
            self.h = min(2.0 / n, 1.0 / m)
            self.rule = {"npts": 3}
            spaces = self.fesp
        else:  # lid-driven cavity
            mesh = E.T6block(1.0, 1.0, n, n)
            pmesh = E.T6toT3(mesh)
            self.fesp = E.FESpace(float, mesh, E.FEH1_T6(), 2)
            self.pfesp = E.FESpace(float, pmesh, E.FEH1_T3(), 1)
            self.fixed = _on_boundary(mesh.xy)
            wall = np.nonzero(self.fixed)[0] + 1
            lid = np.nonzero(mesh.xy[:, 1] == 1.0)[0] + 1
            E.setebc(self.fesp, 0, wall, 1, 0.0)
            E.setebc(self.fesp, 0, wall, 2, 0.0)
            E.setebc(self.fesp, 0, lid, 1, 1.0)
            E.setebc(self.pfesp, 0, 1, 1, 0.0)
            E.numberdofs([self.fesp, self.pfesp])
            self.h = 1.0 / n
            self.rule = {"npts": 3}
            spaces = [self.fesp, self.pfesp]
        self.mesh = mesh
        self.physics = {"elasticity": N.ELFEL_ELASTICITY, "stokes": N.ELFEL_STOKES}.get(problem, N.ELFEL_HEAT)
        both = spaces if isinstance(spaces, list) else [spaces]
        self.ndofs = sum(E.ndofs(s) for s in both)
        self.nu = sum(E.nunknowns(s) for s in both)
        self.T0 = np.zeros(self.ndofs)
        E.gathersysvec(self.T0, spaces)
        self.elit = E.FEIterator(self.fesp)
        self.qpit = E.QPIterator(self.fesp, self.rule)
        self.pelit = E.FEIterator(self.pfesp) if self.pfesp is not None else None
        self.dofs = self.elit.eldofs_table()
        self.pdofs = self.pelit.eldofs_table() if self.pelit is not None else None

    def coords(self, rng):
        """The mesh's coordinates with the interior vertices moved by +-0.2h, midside nodes kept at the midpoints."""
        mesh = self.mesh
        xy = mesh.xy.copy()
        nv = 3 if mesh.etype == "T6" else mesh.nodes_per_elem
        move = np.zeros(mesh.nnodes, dtype=bool)
        move[mesh.conn[:, :nv].ravel() - 1] = True
        move &= ~self.fixed
        k = int(move.sum())
        xy[move] += rng.uniform(-0.2 * self.h, 0.2 * self.h, size=(k, mesh.sdim))
        if mesh.nodes_per_elem == 6:
            c = mesh.conn - 1
            for a in range(3):
                xy[c[:, 3 + a]] = 0.5 * (xy[c[:, a]] + xy[c[:, (a + 1) % 3]])
        return xy

    def coefficients(self, rng):
        """Conductivity, body force or viscosity of one assembly."""
        if self.problem == "elasticity":
            return rng.uniform(-0.1, 0.1, size=(self.mesh.nel, 2))
        if self.problem == "stokes":
            return float(rng.uniform(0.5, 2.0))
        return np.exp(rng.uniform(math.log(0.5), math.log(2.0), self.mesh.nel))


@functools.lru_cache(maxsize=2)
def _problem(problem, n):
    return Problem(problem, n)


def _data(case, seed):
    """(problem, jittered coordinates, coefficients) of a case and a seed."""
    P = _problem(case["problem"], case["n"])
    rng = np.random.default_rng([seed, case["n"]])
    return P, P.coords(rng), P.coefficients(rng)


def _pinned(a):
    """A page-locked copy of an array, as an array."""
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _pinned_empty(n, dtype):
    return torch.empty(max(int(n), 1), dtype=dtype, pin_memory=True).numpy()


def _requests(case, seed):
    """The serving stream's distribution on grids up to case["n"] cells: (element, cells, kappa, Q) each; the
    meshes come from the case, the coefficients from the seed."""
    g = np.random.default_rng(case["mix"])
    k = case["count"]
    cells = np.rint(np.exp(g.uniform(math.log(16.0), math.log(float(case["n"])), k))).astype(int)
    t6 = g.random(k) < 0.5
    r = np.random.default_rng(seed)
    return [("T6" if t6[i] else "T3", int(cells[i]), float(r.uniform(0.5, 2.0)), float(r.uniform(-10.0, -1.0)))
            for i in range(k)]


# ------------------------------------------------------------------ state
def _resident(P, xy, coef):
    """A system set up on the device with these coordinates, assembled once."""
    am = E.start(E.SysmatAssemblerGPU(), P.ndofs, P.ndofs)
    am.setup(P.physics, P.elit, P.qpit, P.pelit, P.ndofs)
    am.set_geometry(xy)
    _assemble(am, P, coef)
    return am


def _assemble(am, P, coef):
    if P.problem == "elasticity":
        am.elasticity(1.0, 0.3, True, coef)
    elif P.problem == "stokes":
        am.stokes(coef)
    else:
        am.heat(coef, Q)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return {"case": case, "requests": _requests(case, seed),
                "server": E.HeatServer("pcg32_ir", max_active=64, rtol=RTOL)}
    P, xy, coef = _data(case, seed)
    s = {"case": case, "P": P, "coef": coef if isinstance(coef, float) else _pinned(coef)}
    if kind in ("reassemble", "solve"):
        s["am"] = _resident(P, xy, coef)
        if kind == "reassemble":
            s["nzval"] = _pinned_empty(_sizes(case["problem"], case["n"])[-1], torch.float64)
            s["F"] = _pinned_empty(P.ndofs, torch.float64)
        return s
    if kind == "script":
        s["mesh"] = E.Mesh(P.mesh.etype, P.mesh.conn, xy)
        return s
    if kind == "coo":
        s["I"] = _pinned(np.repeat(P.dofs[:, None, :], P.dofs.shape[1], axis=1).ravel())  # rows, i fastest
        s["J"] = _pinned(np.repeat(P.dofs[:, :, None], P.dofs.shape[1], axis=2).ravel())
        s["V"] = _pinned(np.random.default_rng([seed, 1]).standard_normal(s["I"].size))
    else:  # assemble_csc: the tables of the two spaces in page-locked memory
        for k, a in (("conn", P.mesh.conn), ("xy", xy), ("dofs", P.dofs)):
            s[k] = _pinned(a)
        if P.pelit is not None:
            s["pconn"], s["pxy"], s["pdofs"] = _pinned(P.pfesp.mesh.conn), _pinned(P.pfesp.mesh.xy), _pinned(P.pdofs)
    ctx = s["ctx"] = E.default_context()
    h = ctypes.c_void_p()
    ctx.check(ctx.lib.elfel_sysmat_create(ctx.h, ctypes.byref(h)))
    s["h"] = _Owned(ctx, h)
    nnz = _sizes(case["problem"], case["n"])[-1]
    s["colptr"] = _pinned_empty(P.ndofs + 1, torch.int64)
    s["rowval"] = _pinned_empty(nnz, torch.int64)
    s["nzval"] = _pinned_empty(nnz, torch.float64)
    s["F"] = _pinned_empty(P.ndofs, torch.float64)
    return s


class _Owned:
    """An elfel_sysmat handle destroyed with the state that holds it."""

    def __init__(self, ctx, h):
        self.ctx, self.h = ctx, h

    def __del__(self):
        if getattr(self.ctx, "h", None):
            self.ctx.lib.elfel_sysmat_destroy(self.h)


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s["case"]["kind"]
    if kind == "reassemble":
        am, ctx = s["am"], s["am"].ctx
        _assemble(am, s["P"], s["coef"])
        ctx.check(ctx.lib.elfel_sysmat_csc(am._hd.h, None, None, N.ptr(s["nzval"])))
        ctx.check(ctx.lib.elfel_sysmat_rhs(am._hd.h, N.ptr(s["F"])))
        return {"nzval": s["nzval"], "F": s["F"]}
    if kind == "assemble_csc":
        return _run_assemble_csc(s)
    if kind == "coo":
        ctx, h, P = s["ctx"], s["h"].h, s["P"]
        L = ctx.lib
        nnz = ctypes.c_int64()
        ctx.check(L.elfel_sysmat_start(h, P.ndofs, P.ndofs))
        ctx.check(L.elfel_sysmat_assemble_coo(h, N.ptr(s["I"], N._i64p), N.ptr(s["J"], N._i64p), N.ptr(s["V"]),
                                              s["V"].size))
        ctx.check(L.elfel_sysmat_finish(h, ctypes.byref(nnz)))
        ctx.check(L.elfel_sysmat_csc(h, N.ptr(s["colptr"], N._i64p), N.ptr(s["rowval"], N._i64p), N.ptr(s["nzval"])))
        return {"colptr": s["colptr"], "rowval": s["rowval"], "nzval": s["nzval"]}
    if kind == "script":
        return _run_script(s)
    if kind == "solve":
        P, am = s["P"], s["am"]
        _assemble(am, P, s["coef"])
        T = P.T0.copy()
        E.solve(T, am, None, P.nu, method=s["case"]["method"], rtol=RTOL)
        return {"T": T}
    srv = s["server"]
    ids = [srv.submit(E.heat_request(et, n, kappa=k, Q=q, keep_solution=True)) for et, n, k, q in s["requests"]]
    srv.drain()
    return [srv.solution(i) for i in ids]


def _run_assemble_csc(s):
    P, ctx, h = s["P"], s["ctx"], s["h"].h
    L, mesh = ctx.lib, P.mesh
    ip = lambda a: N.ptr(a, N._i64p)  # noqa: E731
    u = N.Space(mesh.nodes_per_elem, P.fesp.nfecopies, mesh.nel, mesh.nnodes, ip(s["conn"]), N.ptr(s["xy"]), ip(s["dofs"]))
    p = N.Space()
    if P.pelit is not None:
        pm = P.pfesp.mesh
        p = N.Space(3, 1, pm.nel, pm.nnodes, ip(s["pconn"]), N.ptr(s["pxy"]), ip(s["pdofs"]))
    qr = P.qpit.quadr
    pc, w = N.f64(qr.param_coords), N.f64(qr.weights)
    shape = {"Q4": N.ELFEL_SHAPE_Q4, "T4": N.ELFEL_SHAPE_T4}.get(P.problem, N.ELFEL_SHAPE_TRIANGLE)
    d = N.FusedDesc(P.physics, qr.npts, N.ptr(pc), N.ptr(w), P.ndofs, u, p, shape, mesh.sdim)
    ctx.check(L.elfel_fused_setup(h, ctypes.byref(d)))
    if P.problem == "elasticity":
        ctx.check(L.elfel_fused_elasticity(h, 1.0, 0.3, 1, N.ptr(s["coef"]), None, 0, None))
    elif P.problem == "stokes":
        ctx.check(L.elfel_fused_stokes(h, s["coef"]))
    else:
        ctx.check(L.elfel_fused_heat(h, N.ptr(s["coef"]), Q))
    ctx.check(L.elfel_sysmat_csc(h, ip(s["colptr"]), ip(s["rowval"]), N.ptr(s["nzval"])))
    ctx.check(L.elfel_sysmat_rhs(h, N.ptr(s["F"])))
    return {"colptr": s["colptr"], "rowval": s["rowval"], "nzval": s["nzval"], "F": s["F"]}


def _run_script(s):
    """test/test_heat.jl:89-111 line by line, on the device assembler."""
    P = s["P"]
    mesh = s["mesh"]
    fesp = E.FESpace(float, mesh, type(P.fesp.fe)())
    bn = np.nonzero(P.fixed)[0] + 1
    E.setebc(fesp, 0, bn, 1, _tempf(mesh.xy[bn - 1]))
    E.numberdofs(fesp)
    n, nu = E.ndofs(fesp), E.nunknowns(fesp)
    am = E.start(E.SysmatAssemblerGPU(), n, n)
    E.assemble_heat(am, E.FEIterator(fesp), E.QPIterator(fesp, P.rule), s["coef"], Q)
    T = np.zeros(n)
    E.gathersysvec(T, fesp)
    E.solve(T, am, None, nu, method=s["case"]["method"], rtol=RTOL)
    E.scattersysvec(fesp, T)
    return {"T": T}


# ------------------------------------------------------------------ work
def _sizes(problem, n):
    """(elements, nodes, DOFs, element DOFs, nodes per element, coordinates per node, nonzeros of K)."""
    if problem == "T3":
        v, e = (n + 1) ** 2, 3 * n * n + 2 * n
        return 2 * n * n, v, v, 3, 3, 2, v + 2 * e
    if problem == "Q4":
        v = (n + 1) ** 2
        return n * n, v, v, 4, 4, 2, (3 * n + 1) ** 2
    if problem == "T4":
        v = (n + 1) ** 3
        edges = 3 * n * (n + 1) ** 2 + 3 * n * n * (n + 1) + n ** 3
        return 6 * n ** 3, v, v, 4, 4, 3, v + 2 * edges
    m = max(1, n // 2) if problem == "elasticity" else n
    nel, vert, edge = 2 * n * m, (n + 1) * (m + 1), 3 * n * m + n + m
    nodes = vert + edge
    # node pairs sharing an element: the ordered pairs of each triangle, those on an inner edge counted once
    pairs = 36 * nel - 9 * (edge - 2 * (n + m)) - _inner_vertex_overlap(n, m)
    if problem == "T6":
        return nel, nodes, nodes, 6, 6, 2, pairs
    if problem == "elasticity":
        return nel, nodes, 2 * nodes, 12, 6, 2, 4 * pairs
    return nel, nodes, 2 * nodes + vert, 15, 6, 2, 4 * pairs + 2 * 2 * _p2p1_pairs(n, m)


def _inner_vertex_overlap(n, m):
    """What the count over triangles less that over inner edges still counts too often at vertices."""
    inc = 3 * 2 * n * m  # (vertex, triangle) incidences
    edge_inc = 2 * (3 * n * m + n + m - 2 * (n + m))  # (vertex, inner edge) incidences
    return inc - edge_inc - (n + 1) * (m + 1)


def _p2p1_pairs(n, m):
    """Pairs (T6 node, vertex) that share a triangle."""
    inner = 3 * n * m + n + m - 2 * (n + m)
    return 18 * 2 * n * m - 6 * inner - _inner_vertex_overlap(n, m)


#: FP64 operations of one element's matrix and vector in the tensor form, about.
_ELEMENT_FLOPS = {"T3": 40, "T6": 90, "Q4": 260, "T4": 110, "elasticity": 620, "stokes": 260}


def work(case):
    kind = case["kind"]
    if kind == "serve":
        b = f = 0
        for et, n, _, _ in _requests(case, 0):
            nel, nodes, ndofs, _, nn, _, nnz = _sizes(et, n)
            b += nel * (4 * nn + 8) + 16 * nodes + 12 * nnz + 24 * ndofs
            f += nel * _ELEMENT_FLOPS[et] + 2 * nnz
        return {"bytes": b, "flops": f}
    p = case["problem"]
    nel, nodes, ndofs, nedof, nn, sdim, nnz = _sizes(p, case["n"])
    coef = 16 * nel if p == "elasticity" else 0 if p == "stokes" else 8 * nel
    tables = 8 * sdim * nodes + 4 * nn * nel + coef
    flops = nel * _ELEMENT_FLOPS[p]
    if kind == "reassemble":  # resident tables and coefficients in, values and F out
        return {"bytes": tables + 8 * nnz + 8 * ndofs, "flops": flops}
    if kind == "assemble_csc":  # 64-bit tables in, 64-bit CSC and F out
        return {"bytes": 8 * sdim * nodes + 8 * (nn + nedof) * nel + coef + 16 * nnz + 16 * ndofs, "flops": flops}
    if kind == "coo":
        return {"bytes": 24 * nedof * nedof * nel + 16 * nnz + 8 * ndofs, "flops": nedof * nedof * nel}
    # script and solve: K built and read once, F, T in and out (the iterations are the solver's choice)
    return {"bytes": tables + 20 * nnz + 32 * ndofs, "flops": flops + 2 * nnz}


# ------------------------------------------------------------------ exact
# The same problems in plain torch, 64 bits: element matrices by quadrature,
# duplicates summed after a sort, systems solved by LU or by conjugate
# gradients restarted until the residual no longer falls.
_TRI3 = ([[1 / 6, 1 / 6], [2 / 3, 1 / 6], [1 / 6, 2 / 3]], [1 / 6] * 3)
_G = 1 / math.sqrt(3.0)
_SQUARE4 = ([[-_G, -_G], [_G, -_G], [-_G, _G], [_G, _G]], [1.0] * 4)
_TET1 = ([[0.25, 0.25, 0.25]], [1 / 6])


def _basis(etype, p):
    """Values and parametric gradients at the point p."""
    if etype == "T3":
        r, s = p
        return [1 - r - s, r, s], [[-1, -1], [1, 0], [0, 1]]
    if etype == "T6":
        r, s = p
        t = 1 - r - s
        return ([t * (2 * t - 1), r * (2 * r - 1), s * (2 * s - 1), 4 * r * t, 4 * r * s, 4 * s * t],
                [[1 - 4 * t, 1 - 4 * t], [4 * r - 1, 0], [0, 4 * s - 1], [4 * (t - r), -4 * r], [4 * s, 4 * r],
                 [-4 * s, 4 * (t - s)]])
    if etype == "Q4":
        x, y = p
        c = [(-1, -1), (1, -1), (1, 1), (-1, 1)]
        return ([0.25 * (1 + a * x) * (1 + b * y) for a, b in c],
                [[0.25 * a * (1 + b * y), 0.25 * b * (1 + a * x)] for a, b in c])
    r, s, u = p
    return [1 - r - s - u, r, s, u], [[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]]


def _elements(problem, conn, xy, coef, q_source=Q):
    """(ke, fe, kup) of all elements; kup for Stokes only."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda a: torch.as_tensor(np.asarray(a), device=dev)  # noqa: E731
    etype = problem if problem in ("T3", "Q4", "T4") else "T6"
    pts, ws = _SQUARE4 if etype == "Q4" else _TET1 if etype == "T4" else _TRI3
    X = t(xy)[t(conn) - 1]  # nel x nn x sdim
    nel, nn, sd = X.shape
    comp = 2 if problem in ("elasticity", "stokes") else 1
    ke = torch.zeros(nel, nn * comp, nn * comp, dtype=torch.float64, device=dev)
    fe = torch.zeros(nel, nn * comp, dtype=torch.float64, device=dev)
    kup = torch.zeros(nel, 12, 3, dtype=torch.float64, device=dev) if problem == "stokes" else None
    c = t(coef) if problem != "stokes" else coef
    if problem == "elasticity":
        f = 1.0 / (1.3 * 0.4)
        D = t([[f * 0.7, f * 0.3, 0.0], [f * 0.3, f * 0.7, 0.0], [0.0, 0.0, f * 0.2]])
    for p, w in zip(pts, ws):
        Nq, Gq = _basis(etype, p)
        Nq, Gq = t(np.array(Nq, dtype=float)), t(np.array(Gq, dtype=float))
        J = torch.einsum("enx,na->exa", X, Gq)
        det = torch.linalg.det(J)
        g = torch.matmul(Gq, torch.linalg.inv(J))  # nel x nn x sdim
        if problem == "elasticity":
            B = torch.zeros(nel, 3, nn, 2, dtype=torch.float64, device=dev)
            B[:, 0, :, 0] = g[:, :, 0]
            B[:, 1, :, 1] = g[:, :, 1]
            B[:, 2, :, 0] = g[:, :, 1]
            B[:, 2, :, 1] = g[:, :, 0]
            B = B.reshape(nel, 3, 2 * nn)
            ke += torch.matmul(B.transpose(1, 2), torch.matmul(D, B)) * (w * det)[:, None, None]
            fe += (Nq[None, :, None] * c[:, None, :] * (w * det)[:, None, None]).reshape(nel, 2 * nn)
        elif problem == "stokes":
            L = torch.matmul(g, g.transpose(1, 2)) * (c * w * det)[:, None, None]
            ke[:, 0::2, 0::2] += L
            ke[:, 1::2, 1::2] += L
            Np = t(np.array(_basis("T3", p)[0], dtype=float))
            kup -= (w * det)[:, None, None] * g.reshape(nel, 12)[:, :, None] * Np[None, None, :]
        else:
            ke += torch.matmul(g, g.transpose(1, 2)) * (c * w * det)[:, None, None]
            fe += Nq[None, :] * (q_source * w * det)[:, None]
    return ke, fe, kup


def _sum_csc(rows, cols, vals, n):
    """(row, col, value) of the distinct entries, column by column, duplicates added."""
    key, order = torch.sort(cols * n + rows)
    u, inv = torch.unique_consecutive(key, return_inverse=True)
    out = torch.zeros(u.numel(), dtype=torch.float64, device=vals.device).index_add_(0, inv, vals[order])
    return u % n, u // n, out


def _system(problem, conn, xy, dofs, pdofs, n, coef, q_source=Q):
    """(row, col, value) of K in CSC order and F."""
    ke, fe, kup = _elements(problem, conn, xy, coef, q_source)
    d = torch.as_tensor(dofs, device=ke.device) - 1
    nd = d.shape[1]
    R, C, V = [d[:, :, None].expand(-1, nd, nd)], [d[:, None, :].expand(-1, nd, nd)], [ke]
    if kup is not None:
        p = torch.as_tensor(pdofs, device=ke.device) - 1
        ru, cp = d[:, :, None].expand(-1, 12, 3), p[:, None, :].expand(-1, 12, 3)
        R += [ru, cp]
        C += [cp, ru]
        V += [kup, kup]
    flat = [torch.cat([x.reshape(-1) for x in v]) for v in (R, C, V)]
    r, c, v = _sum_csc(*flat, n)
    F = torch.zeros(n, dtype=torch.float64, device=ke.device).index_add_(0, d.reshape(-1), fe.reshape(-1))
    return r, c, v, F


def _solve_exact(r, c, v, F, T0, nu, definite):
    n = F.numel()
    T = torch.as_tensor(T0, device=v.device).clone()
    K = torch.sparse_coo_tensor(torch.stack([r, c]), v, (n, n)).coalesce()
    b = (F - torch.mv(K, T))[:nu]
    ff = (r < nu) & (c < nu)
    A = torch.sparse_coo_tensor(torch.stack([r[ff], c[ff]]), v[ff], (nu, nu)).coalesce()
    if nu <= 12000:
        D = A.to_dense()
        x = torch.linalg.solve(D, b)
        x = x + torch.linalg.solve(D, b - torch.mv(D, x))
    elif definite:
        x = _cg(A.to_sparse_csr(), A, b)
    else:
        return None
    T[:nu] += x
    return T.cpu().numpy()


def _cg(A, coo, b):
    idx = coo.indices()
    diag = coo.values()[idx[0] == idx[1]]
    x = torch.zeros_like(b)
    best = None
    for _ in range(4):
        r = b - torch.mv(A, x)
        size = float(r.norm())
        if best is not None and size > 0.5 * best[0]:
            x = best[1] if size > best[0] else x
            break
        best = (size, x.clone())
        z = r / diag
        p, rz, stop = z, torch.dot(r, z), 1e-13 * size
        for k in range(40000):
            q = torch.mv(A, p)
            a = rz / torch.dot(p, q)
            x = x + a * p
            r = r - a * q
            if k % 64 == 0 and float(r.norm()) <= stop:
                break
            z = r / diag
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return [_served_exact(*q) for q in _requests(case, seed)]
    P, xy, coef = _data(case, seed)
    if kind == "coo":
        d = torch.as_tensor(P.dofs, device="cuda" if torch.cuda.is_available() else "cpu") - 1
        nd = d.shape[1]
        V = torch.as_tensor(np.random.default_rng([seed, 1]).standard_normal(d.numel() * nd), device=d.device)
        _, _, v = _sum_csc(d[:, None, :].expand(-1, nd, nd).reshape(-1), d[:, :, None].expand(-1, nd, nd).reshape(-1),
                           V, P.ndofs)
        return {"colptr": None, "rowval": None, "nzval": v.cpu().numpy()}
    r, c, v, F = _system(P.problem, P.mesh.conn, xy, P.dofs, P.pdofs, P.ndofs, coef)
    if kind == "reassemble":
        return {"nzval": v.cpu().numpy(), "F": F.cpu().numpy()}
    if kind == "assemble_csc":
        return {"colptr": None, "rowval": None, "nzval": v.cpu().numpy(), "F": F.cpu().numpy()}
    return {"T": _solve_exact(r, c, v, F, P.T0, P.nu, P.problem != "stokes")}


def _served_exact(etype, n, kappa, q):
    P = _problem(etype, n)
    r, c, v, F = _system(etype, P.mesh.conn, P.mesh.xy, P.dofs, None, P.ndofs, np.full(P.mesh.nel, kappa), q)
    return _solve_exact(r, c, v, F, P.T0, P.nu, True)
