"""The one-launch Krylov iterations (krylov.cu) at the edges of their ranges (GPU).

A system runs in a cluster of 1 to 16 blocks, or in a grid of one block per SM,
by its number of unknowns; the sizes sit on both sides of every line: a partly
filled slice, the cluster sizes, cluster / grid, three and two barriers an
iteration, matrix in shared memory or not, 16-bit and 32-bit columns, systems
too large for any group.  Every solution is compared with the oracle's direct
solve (relative, 2-norm).

Tolerance: the matrices have condition number at most 9 (eigenvalues of modulus
1 to 9), so a relative residual of 1e-11 leaves ||x - x0|| <= 9e-11 ||x0|| in
the 2-norm; 1e-10 with the direct solution's own rounding.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10


def laplacian(n, shuffle=None):
    """The leading n x n block of I + the 5-point Laplacian of a square grid."""
    import scipy.sparse as sp

    m = int(np.ceil(np.sqrt(n)))
    L = sp.diags([-np.ones(m - 1), 2.0 * np.ones(m), -np.ones(m - 1)], [-1, 0, 1])
    A = (sp.identity(m * m) + sp.kron(sp.identity(m), L) + sp.kron(L, sp.identity(m))).tocsr()[:n, :n]
    if shuffle is not None:
        p = np.random.default_rng(shuffle).permutation(n)
        A = A[p][:, p]
    return A.tocsc()


def solve_both(E, O, A, nu, method, ctx=None):
    n = A.shape[0]
    rng = np.random.default_rng(n)
    F = rng.standard_normal(n)
    T = np.zeros(n)
    T[nu:] = rng.standard_normal(n - nu)
    T0 = O.solve_lifted(A, F, T.copy(), nu)
    st = E.solve(T, A, F, nu, method=method, rtol=1e-11, ctx=ctx)
    assert st["converged"] and st["relres"] <= 1e-11
    assert np.linalg.norm(T[:nu] - T0[:nu]) <= TOL * np.linalg.norm(T0[:nu]), (n, nu, method)
    return st


SIZES = [1, 31, 32, 33, 64, 65, 129, 257, 513, 1024, 1025, 4097, 16384, 16385, 32768, 32769, 65536, 65537, 262145]


@pytest.mark.parametrize("method", ["pcg64", "pcg32_ir"])
@pytest.mark.parametrize("nu", SIZES)
def test_sizes(E, O, gpu, nu, method):
    solve_both(E, O, laplacian(nu + 3), nu, method)


@pytest.mark.parametrize("method", ["pcg64", "pcg32_ir"])
@pytest.mark.parametrize("nu", [2049, 40000, 70000])
def test_wide_columns(E, O, gpu, nu, method):
    """Shuffled numbering: 32-bit columns beyond 32k, and blocks that gather from every other block."""
    solve_both(E, O, laplacian(nu, shuffle=3), nu, method)


@pytest.mark.parametrize("method", ["pcg64", "pcg32_ir"])
@pytest.mark.parametrize("nu", [1025, 20001, 70001])
def test_same_iterations_as_graphs(E, O, gpu, monkeypatch, nu, method):
    """The graph of three kernels (ELFEL_ONE_LAUNCH=0) runs the same recurrence:
    the same number of iterations, give or take what rounding moves at the
    stopping line (a few), and the same answer."""
    A = laplacian(nu)
    one = solve_both(E, O, A, nu, method)
    monkeypatch.setenv("ELFEL_ONE_LAUNCH", "0")
    ctx = E.Context(0)
    many = solve_both(E, O, A, nu, method, ctx)
    assert abs(one["iterations"] - many["iterations"]) <= 3


@pytest.mark.parametrize("method", ["minres64", "minres32_ir"])
@pytest.mark.parametrize("nu", [1, 33, 1025, 16385, 32769, 70001])
def test_minres_sizes(E, O, gpu, nu, method):
    """An indefinite system: I + Laplacian on two rows of three, its negative on the third."""
    import scipy.sparse as sp

    n2 = nu // 3
    order = np.argsort(np.argsort(np.arange(nu) % 3 == 2, kind="stable"))
    parts = [laplacian(nu - n2)] + ([-laplacian(n2)] if n2 else [])
    B = sp.block_diag(parts).tocsr()[order][:, order].tocsc()
    F = np.random.default_rng(nu).standard_normal(nu)
    T0 = O.solve_lifted(B, F, np.zeros(nu), nu)
    T = np.zeros(nu)
    st = E.solve(T, B, F, nu, method=method, rtol=1e-11, maxit=20000)
    assert st["converged"] and st["relres"] <= 1e-11
    assert np.linalg.norm(T - T0) <= TOL * np.linalg.norm(T0)


@pytest.mark.parametrize("nu", [500, 20000])
def test_iteration_limit(E, gpu, nu):
    A = laplacian(nu)
    for method in ("pcg64", "pcg32_ir", "minres64"):
        with pytest.raises(E.NotConverged) as e:
            E.solve(np.zeros(nu), A, np.ones(nu) + np.arange(nu) % 7, nu, method=method, rtol=1e-11, maxit=4)
        assert "after 4 iterations" in str(e.value)


def test_two_contexts_at_once(E, O, gpu):
    """Grid groups of two contexts, launched from two threads: both end, with the answers they have alone."""
    import threading

    A = laplacian(20001)
    F = np.random.default_rng(1).standard_normal(A.shape[0])
    T0 = O.solve_lifted(A, F, np.zeros(A.shape[0]), A.shape[0])
    errs = []

    def work():
        try:
            ctx = E.Context(0)
            a = E.start(E.SysmatAssemblerSparse(0.0, ctx=ctx), *A.shape)
            c = A.tocoo()
            a._chunks.append((c.row.astype(np.int64) + 1, c.col.astype(np.int64) + 1, c.data.astype(np.float64)))
            E.finish(a)
            for _ in range(20):
                T = np.zeros(A.shape[0])
                E.solve(T, a, F, A.shape[0], method="pcg64", rtol=1e-11)
                errs.append(float(np.linalg.norm(T - T0) / np.linalg.norm(T0)))
        except Exception as e:  # reported by the assertion below
            errs.append(e)

    th = [threading.Thread(target=work) for _ in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert len(errs) == 40 and all(isinstance(e, float) and e <= TOL for e in errs), errs[:4]


BATCH = {"pcg32_ir": [1, 33, 2048, 2049, 4097, 8193, 16385, 32768, 40960, 40993],
         "pcg64": [1, 33, 1024, 1025, 2049, 4097, 8193, 16384, 20480, 20513]}


@pytest.mark.parametrize("method", sorted(BATCH))
def test_batched_clusters(E, O, gpu, method):
    """Batched systems on both sides of every cluster size (1 to 16 blocks) and
    beyond the largest, one of them with 32-bit columns: the direct solution
    within TOL, and the same bits alone and in the mix."""
    probs = []
    for i, n in enumerate(BATCH[method] + [36000 if method == "pcg32_ir" else 20000]):
        A = laplacian(n, shuffle=5 if i == len(BATCH[method]) else None)
        c = A.tocoo()
        a = E.start(E.SysmatAssemblerSparse(), n, n)
        a._chunks.append((c.row.astype(np.int64) + 1, c.col.astype(np.int64) + 1, c.data.astype(np.float64)))
        E.finish(a)
        F = np.random.default_rng(n).standard_normal(n)
        probs.append((A, a, F))

    def run(which):
        b = E.BatchSolver(method, capacity=len(which))
        slots = [b.add(probs[i][1], np.zeros(probs[i][0].shape[0]), probs[i][0].shape[0], F=probs[i][2], rtol=1e-11)
                 for i in which]
        out = b.run()
        b.close()
        return [out[s] for s in slots]

    mixed = run(list(range(len(probs))))
    for i, (A, a, F) in enumerate(probs):
        T, st = mixed[i]
        assert st["converged"] and st["relres"] <= 1e-11
        T0 = O.solve_lifted(A, F, np.zeros(A.shape[0]), A.shape[0])
        assert np.linalg.norm(T - T0) <= TOL * np.linalg.norm(T0), A.shape
        (Ta, sta), = run([i])
        assert np.array_equal(T, Ta) and st["iterations"] == sta["iterations"], A.shape
