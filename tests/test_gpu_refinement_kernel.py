"""The FP32 refinement with its residual replacements inside the iteration kernel, cluster and grid (run_ir) (GPU).

Against the graphs of three kernels with the replacements on the host
(ELFEL_ONE_LAUNCH=0): both stop at a relative residual of 1e-10, so with
condition numbers of at most 9 (I + the five-point Laplacian) each solution is
within 9e-10 of the exact one in the 2-norm and the two within 2e-9.
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def laplacian(n):
    m = int(np.ceil(np.sqrt(n)))
    L = sp.diags([-np.ones(m - 1), 2.0 * np.ones(m), -np.ones(m - 1)], [-1, 0, 1])
    return (sp.identity(m * m) + sp.kron(sp.identity(m), L) + sp.kron(L, sp.identity(m))).tocsr()[:n, :n].tocsc()


@pytest.mark.parametrize("n", [1, 32, 33, 257, 1025, 8193, 32768, 32769, 70001, 400000])
@pytest.mark.parametrize("scale", [1.0, 1e-30, 1e25])
def test_against_graphs(E, gpu, monkeypatch, n, scale):
    A = laplacian(n)
    F = scale * np.random.default_rng(n).standard_normal(n)
    out = []
    for on in ("1", "0"):
        monkeypatch.setenv("ELFEL_ONE_LAUNCH", on)
        T = np.zeros(n)
        st = E.solve(T, A, F, n, method="pcg32_ir", rtol=1e-10, ctx=E.Context(0))
        assert st["converged"] and st["relres"] <= 1e-10
        out.append(T)
    assert np.linalg.norm(out[0] - out[1]) <= 2e-9 * np.linalg.norm(out[1])


def test_more_iterations_than_a_launch(E, gpu):
    """A 1-D Laplacian whose refinement needs more than the 4096 iterations of one launch."""
    n = 3000
    A = sp.diags([-np.ones(n - 1), 2.0 * np.ones(n), -np.ones(n - 1)], [-1, 0, 1]).tocsc()
    F = np.random.default_rng(0).standard_normal(n)
    T = np.zeros(n)
    st = E.solve(T, A, F, n, method="pcg32_ir", rtol=1e-8)
    assert st["converged"] and st["iterations"] > 4096
    assert np.linalg.norm(F - A @ T) <= 1.01e-8 * np.linalg.norm(F)


@pytest.mark.parametrize("maxit", [1, 7])
def test_iteration_limit(E, gpu, maxit):
    A = laplacian(500)
    T = np.zeros(500)
    with pytest.raises(E.ElfelError):
        E.solve(T, A, np.ones(500) + np.arange(500), 500, method="pcg32_ir", rtol=1e-12, maxit=maxit)
