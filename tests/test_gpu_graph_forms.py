"""The iterations in graphs of small kernels, where the one-launch forms do not reach (GPU).

Systems beyond the limits of the clusters and grids, and every system with
ELFEL_ONE_LAUNCH=0, iterate in the graphs: batches of several such systems (the
same bits alone, in any mix and whenever they join, and in the persistent form),
MINRES, and the hand-over between the forms on both sides of the limits.  Also
here: one-launch MINRES on numberings whose columns come from everywhere.

Solutions: 1e-8 of the oracle's direct solve for the heat systems (relative
residual 1e-10).  The five-point systems have condition numbers of at most 9, so
a relative residual of 1e-11, formed on the host, leaves a relative error of 9e-11.
"""
import numpy as np
import pytest
import scipy.sparse as sp

from problems import heat_oracle, heat_space

pytestmark = pytest.mark.gpu

SMALL = [("T3", 9, 1), ("T6", 14, 2), ("T3", 48, 3), ("T6", 30, 4), ("T3", 3, 5), ("T6", 41, 6)]


def make(E, ctx, etype, n, seed):
    mesh = E.jitter((E.T3block if etype == "T3" else E.T6block)(1.0, 1.0, n, n), 0.1 / n, seed=seed)
    fesp = heat_space(E, mesh, E.FEH1_T3() if etype == "T3" else E.FEH1_T6())
    nd, nu = E.ndofs(fesp), E.nunknowns(fesp)
    kappa = np.random.default_rng(seed).uniform(0.5, 2.0, mesh.nel)
    am = E.start(E.SysmatAssemblerGPU(ctx=ctx), nd, nd)
    E.assemble_heat(am, E.FEIterator(fesp), E.QPIterator(fesp, {"npts": 3}), kappa, -6.0)
    T = np.zeros(nd)
    E.gathersysvec(T, fesp)
    return dict(mesh=mesh, fesp=fesp, am=am, T=T, nu=nu, kappa=kappa)


def graphs_ctx(E, monkeypatch):
    monkeypatch.setenv("ELFEL_ONE_LAUNCH", "0")
    return E.Context(0)


def batch(E, ctx, probs, method, graphs=2, capacity=8):
    b = E.BatchSolver(method, capacity=capacity, ctx=ctx)
    slots = [b.add(p["am"], p["T"], p["nu"], rtol=1e-10) for p in probs]
    out = b.run(graphs=graphs)
    b.close()
    return [out[s] for s in slots]


def same(a, b):
    assert np.array_equal(a[0], b[0]) and a[1]["iterations"] == b[1]["iterations"]


# unknowns beyond the largest cluster system (40,960 in FP32, 20,480 in FP64), twice, with small ones beside
LARGE = {"pcg32_ir": [("T6", 104, 7), ("T3", 30, 8), ("T3", 215, 9), ("T6", 20, 10)],
         "pcg64": [("T6", 74, 7), ("T3", 30, 8), ("T3", 150, 9), ("T6", 20, 10)]}


@pytest.mark.parametrize("method", ["pcg32_ir", "pcg64"])
@pytest.mark.parametrize("which", ["small", "large"])
def test_batch_alone_mixed_persistent(E, O, gpu, monkeypatch, method, which):
    ctx = graphs_ctx(E, monkeypatch) if which == "small" else E.Context(0)
    probs = [make(E, ctx, *m) for m in (SMALL if which == "small" else LARGE[method])]
    mixed = batch(E, ctx, probs, method)
    for p, r in zip(probs, mixed):
        assert r[1]["converged"] and r[1]["relres"] <= 1e-10
        K0, F0 = heat_oracle(E, O, p["mesh"], p["fesp"], 3, p["kappa"], -6.0)
        T0 = O.solve_lifted(K0, F0, p["T"].copy(), p["nu"])
        assert np.abs(r[0] - T0).max() <= 1e-8 * np.abs(T0).max()
        same(r, batch(E, ctx, [p], method, capacity=1)[0])
    monkeypatch.setenv("ELFEL_BATCH_PERSIST", "1")
    for r, q in zip(mixed, batch(E, ctx, probs, method)):
        same(r, q)


@pytest.mark.parametrize("method", ["pcg32_ir", "pcg64"])
@pytest.mark.parametrize("which", ["small", "large"])
def test_staggered_joins(E, gpu, monkeypatch, method, which):
    ctx = graphs_ctx(E, monkeypatch) if which == "small" else E.Context(0)
    probs = [make(E, ctx, *m) for m in (SMALL if which == "small" else LARGE[method])]
    ref = batch(E, ctx, probs, method)
    b = E.BatchSolver(method, capacity=4, ctx=ctx)
    pending, slot_of, got = list(range(len(probs))), {}, {}
    while pending or slot_of:
        if pending and len(slot_of) < 4:
            i = pending.pop(0)
            slot_of[b.add(probs[i]["am"], probs[i]["T"], probs[i]["nu"], rtol=1e-10)] = i
        b.step(1)
        for s in b.done():
            got[slot_of.pop(s)] = b.result(s)
    b.close()
    for i, r in enumerate(ref):
        same(got[i], r)


def laplacian(n, shuffle=None):
    m = int(np.ceil(np.sqrt(n)))
    L = sp.diags([-np.ones(m - 1), 2.0 * np.ones(m), -np.ones(m - 1)], [-1, 0, 1])
    A = (sp.identity(m * m) + sp.kron(sp.identity(m), L) + sp.kron(L, sp.identity(m))).tocsr()[:n, :n]
    if shuffle is not None:
        p = np.random.default_rng(shuffle).permutation(n)
        A = A[p][:, p]
    return A


def indefinite(n, shuffle=None):
    """I + Laplacian on two rows of three, its negative on the third."""
    n2 = n // 3
    order = np.argsort(np.argsort(np.arange(n) % 3 == 2, kind="stable"))
    if shuffle is not None:
        order = np.random.default_rng(shuffle).permutation(n)
    return sp.block_diag([laplacian(n - n2)] + ([-laplacian(n2)] if n2 else [])).tocsr()[order][:, order]


def solve(E, ctx, A, method):
    n = A.shape[0]
    c = A.tocoo()
    a = E.start(E.SysmatAssemblerSparse(0.0, ctx=ctx), n, n)
    a._chunks.append((c.row.astype(np.int64) + 1, c.col.astype(np.int64) + 1, c.data.astype(np.float64)))
    E.finish(a)
    F, T = np.random.default_rng(n).standard_normal(n), np.zeros(n)
    st = E.solve(T, a, F, n, method=method, rtol=1e-11, maxit=20000)
    assert st["converged"] and st["relres"] <= 1e-11
    # the host's residual differs from the device's by the rounding of its own sums
    assert np.linalg.norm(F - A @ T) <= 1.01e-11 * np.linalg.norm(F)
    return T, st


@pytest.mark.parametrize("method", ["minres64", "minres32_ir"])
@pytest.mark.parametrize("n", [1, 33, 1025, 16385, 70001])
def test_minres_graphs(E, gpu, monkeypatch, method, n):
    """The four graph kernels of MINRES against the one-launch form: the same recurrence, so nearly as many iterations."""
    A = indefinite(n)
    T1, st1 = solve(E, gpu, A, method)
    T0, st0 = solve(E, graphs_ctx(E, monkeypatch), A, method)
    assert np.linalg.norm(T1 - T0) <= 2e-10 * np.linalg.norm(T0)
    if method == "minres64":
        assert abs(st1["iterations"] - st0["iterations"]) <= 3


@pytest.mark.parametrize("method", ["minres64", "minres32_ir"])
@pytest.mark.parametrize("n", [2049, 40000, 70000])
def test_minres_columns_from_everywhere(E, gpu, method, n):
    solve(E, gpu, indefinite(n, shuffle=3), method)


def most_rows(method):
    """The largest system whose vectors the blocks of the grid hold: 230,400 bytes a block, 12,416 of them
    for the sums; a slice of 32 rows takes its vectors, the gathered one, and 8 bytes."""
    import torch

    sms = min(torch.cuda.get_device_properties(0).multi_processor_count, 160)
    elem, vecs = (8 if method.endswith("64") else 4), (4 if method.startswith("pcg") else 7)
    return sms * ((230400 - 12416) // (32 * (vecs + 1) * elem + 8)) * 32


@pytest.mark.parametrize("method", ["pcg64", "pcg32_ir", "minres64", "minres32_ir"])
@pytest.mark.parametrize("beyond", [0, 1])
def test_both_sides_of_the_limit(E, gpu, method, beyond):
    n = most_rows(method) + beyond
    solve(E, gpu, laplacian(n) if method.startswith("pcg") else indefinite(n), method)
