"""Infinities, NaN and degenerate elements in the closed-form T6 elasticity records (elast_t6_exact_k) (GPU).

The tabulated kernel (a rule whose first weight is larger by 6e-14, which is not
recognised as exact) multiplies every entry of its tables with the element's
values, the zeros too: what is not finite spoils the same entries of K and F in both.
"""
import numpy as np
import pytest

from problems import elasticity_setup

pytestmark = pytest.mark.gpu


def assemble(E, mesh, fesp, off, modulus, bforce):
    q = E.QPIterator(fesp, {"npts": 3})
    if off:
        w = np.array(q.quadr.weights, dtype=float).copy()
        w[0] *= 1.0 + 6e-14
        q.quadr.weights = w
    n = E.ndofs(fesp)
    am = E.start(E.SysmatAssemblerGPU(), n, n)
    E.assemble_elasticity(am, E.FEIterator(fesp), q, modulus, 0.3, True, bforce)
    return E.finish(am), am.rhs().copy()


@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 3), (40, 40)])
@pytest.mark.parametrize("what", ["force nan", "force inf", "one component", "modulus inf", "modulus nan", "flat mesh",
                                  "collapsed element"])
def test_same_entries(E, gpu, nx, ny, what):
    mesh, fesp, bforce, _ = elasticity_setup(E, nx, ny)
    k, modulus = mesh.nel // 2, 3.0
    if what == "force nan":
        bforce[k] = np.nan
    elif what == "force inf":
        bforce[k] = [np.inf, -np.inf]
    elif what == "one component":
        bforce[k, 1] = np.nan
    elif what == "modulus inf":
        modulus = np.inf
    elif what == "modulus nan":
        modulus = np.nan
    elif what == "flat mesh":
        mesh.xy[:, 0] = 0.25
    else:
        mesh.xy[mesh.conn[k] - 1] = mesh.xy[mesh.conn[k, 0] - 1]
    (K1, F1), (K0, F0) = (assemble(E, mesh, fesp, off, modulus, bforce) for off in (False, True))
    assert np.array_equal(K1.indptr, K0.indptr) and np.array_equal(K1.indices, K0.indices)
    if what != "collapsed element":  # (whose neighbours are curved: both take the per-point kernel but on 1 x 1)
        assert not (np.isfinite(K0.data).all() and np.isfinite(F0).all())
    for a, b in ((K1.data, K0.data), (F1, F0)):
        ok = np.isfinite(b)
        assert np.array_equal(np.isfinite(a), ok)
        if ok.any():  # within the two kernels' tolerance for finite systems
            assert np.abs(a[ok] - b[ok]).max() <= 2e-13 * max(np.abs(b[ok]).max(), 1e-300)
