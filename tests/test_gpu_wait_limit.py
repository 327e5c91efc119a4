"""A wait of the one-launch iterations that runs out (GPU): the solve starts again in graphs.

The grid of an iteration kernel needs every SM at once; where another kernel
holds some of them for longer than the limit of its waits, the solve has to end
as it does in graphs.  Here the limit is no poll at all (ELFEL_RUN_SPINS=0): the
first block to arrive gives up, and every other one with it.  Every wait is
bounded, so nothing hangs.  The same graphs from the same start: equal to the
solve with ELFEL_ONE_LAUNCH=0 bit for bit.  Cluster systems (33, 2000) have no
such waits and do not change.
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def laplacian(n):
    m = int(np.ceil(np.sqrt(n)))
    L = sp.diags([-np.ones(m - 1), 2.0 * np.ones(m), -np.ones(m - 1)], [-1, 0, 1])
    return (sp.identity(m * m) + sp.kron(sp.identity(m), L) + sp.kron(L, sp.identity(m))).tocsr()[:n, :n].tocsc()


@pytest.mark.parametrize("method", ["pcg64", "pcg32_ir", "minres64", "minres32_ir"])
@pytest.mark.parametrize("n", [33, 2000, 70001, 400000])
def test_solve_ends_in_graphs(E, gpu, monkeypatch, capfd, n, method):
    A = laplacian(n)
    F = np.random.default_rng(n).standard_normal(n)
    monkeypatch.setenv("ELFEL_TRACE", "1")

    def solve(**env):
        for k in ("ELFEL_ONE_LAUNCH", "ELFEL_RUN_SPINS"):
            monkeypatch.delenv(k, raising=False)
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        ctx = E.Context(0)
        a = E.start(E.SysmatAssemblerSparse(0.0, ctx=ctx), n, n)
        c = A.tocoo()
        a._chunks.append((c.row.astype(np.int64) + 1, c.col.astype(np.int64) + 1, c.data.astype(np.float64)))
        E.finish(a)
        out = []
        for _ in range(2):  # the limit is met again in every solve
            T = np.zeros(n)
            st = E.solve(T, a, F, n, method=method, rtol=1e-11)
            assert st["converged"] and st["relres"] <= 1e-11
            out.append(T)
        return out, capfd.readouterr().err.count("starting again in graphs")

    (one, again), ran_out = solve()
    assert ran_out == 0 and np.array_equal(one, again)
    (late, late2), ran_out = solve(ELFEL_RUN_SPINS="0")
    (graphs, _), none = solve(ELFEL_ONE_LAUNCH="0")
    assert none == 0
    if n <= 2000:
        assert ran_out == 0 and np.array_equal(late, one)
    else:
        assert ran_out == 2
        assert np.array_equal(late, graphs) and np.array_equal(late2, graphs)
