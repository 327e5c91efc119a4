"""The solver's CSR by the symmetric transpose (transpose_sym_k) and, for patterns that are not symmetric, by the pattern builder (GPU).

K = 5 I + the five-point Laplacian has a condition number below 13 / 5, so a
solution with a residual of 1e-12 is within 3e-12 of the exact one; the
tolerance is 1e-11 of the largest value.  Explicit zeros in one triangle leave
the values and make the pattern asymmetric.
"""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

pytestmark = pytest.mark.gpu


def system(n, zeros, rng):
    m = max(1, int(np.ceil(np.sqrt(n))))
    L = sp.kronsum(*[sp.diags([-1.0, 2.0, -1.0], [-1, 0, 1], shape=(m, m))] * 2, format="csr")[:n, :n]
    K = (L + 5.0 * sp.identity(n)).tocoo()
    p = rng.permutation(n)
    I, J, V = p[K.row], p[K.col], K.data
    if zeros:
        i, j = rng.integers(0, n, zeros), rng.integers(0, n, zeros)
        I, J, V = np.r_[I, np.minimum(i, j)], np.r_[J, np.maximum(i, j)], np.r_[V, np.zeros(zeros)]
    return I, J, V


@pytest.mark.parametrize("n", [1, 2, 31, 33, 257, 3000])
@pytest.mark.parametrize("zeros", [0, 1, 500])
@pytest.mark.parametrize("method", ["pcg64", "pcg32_ir", "minres64"])
@pytest.mark.parametrize("data", [0, 1, 5])
def test_solution(E, gpu, n, zeros, method, data):
    rng = np.random.default_rng(n + zeros)
    I, J, V = system(n, zeros, rng)
    nu = max(n - data, 0)
    am = E.start(E.SysmatAssemblerSparse(0.0), n, n)
    for i, j, v in zip(I + 1, J + 1, V):
        E.assemble(am, int(i), int(j), float(v))
    E.finish(am)
    K = sp.coo_matrix((V, (I, J)), shape=(n, n)).tocsc()
    F, T = rng.standard_normal(n), np.zeros(n)
    T[nu:] = rng.standard_normal(n - nu)
    want = T.copy()
    if nu:
        want[:nu] = spl.spsolve(K[:nu, :nu].tocsc(), (F - K @ T)[:nu])
    E.solve(T, am, F, nu, method=method, rtol=1e-12)
    assert np.abs(T - want).max() <= 1e-11 * max(1.0, np.abs(want).max())
